"""An expired wait between the CTAs of a persistent launch (gpu): CUFSP_GRID_WAIT_NS=0 makes the second poll of
a wait that finds nothing give up (among some 100 CTAs and hundreds of waits there always is one), every CTA
leaves, the call returns CUFSP_ERR_CUDA, and the next solve of the same object gives the bits of an undisturbed one."""
import numpy as np
import pytest

from cuda_fsp_b200 import BDFIntegrator, CufspError, FSPMat, KryExpvFSP, MatrixFormat, models

pytestmark = pytest.mark.gpu

MODELS = {
    "registers": lambda: models.toggle((210, 200)),
    "general": lambda: models.mass_action_3(bounds=(70, 60, 40)),  # basis partly in L2
}


@pytest.mark.parametrize("name", MODELS)
@pytest.mark.parametrize("steps_before", [0, 1])
def test_krylov(cuda, monkeypatch, name, steps_before):
    import torch
    m = MODELS[name]()
    A = FSPMat.from_model(m, MatrixFormat.KRONECKER)
    t = 500.0 if name == "registers" else 0.02
    out, stats = [], []
    for expire in (False, True):
        v = torch.as_tensor(m.p0(), device="cuda")
        E = KryExpvFSP(t, A, v, tol=1e-9, coefs=m.coefs(0))
        for _ in range(steps_before):
            E.step()
        if expire:
            monkeypatch.setenv("CUFSP_GRID_WAIT_NS", "0")
            for _ in range(2):
                with pytest.raises(CufspError) as e:
                    E.step()
                assert e.value.name == "CUFSP_ERR_CUDA" and "expired" in str(e.value)
            monkeypatch.delenv("CUFSP_GRID_WAIT_NS")
        stats.append(E.solve())
        out.append(v.cpu().numpy())
    assert stats[0] == stats[1] and stats[0]["n_steps"] > steps_before
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("steps_before", [0, 3])
def test_bdf(cuda, monkeypatch, steps_before):
    import torch
    m = models.gene_expression((1, 1, 1, 60, 70), time_varying=False)
    A = FSPMat.from_model(m, MatrixFormat.KRONECKER)
    p0 = torch.as_tensor(m.p0(), device="cuda")
    out, stats = [], []
    for expire in (False, True):
        p = p0.clone()
        B = BDFIntegrator(A, coefs=m.coefs(0), rtol=1e-8, atol=1e-14)
        B.init(0.0, p0)
        for _ in range(steps_before):
            B.step(0.5, p)
        if expire:
            monkeypatch.setenv("CUFSP_GRID_WAIT_NS", "0")
            with pytest.raises(CufspError) as e:
                B.advance(0.5, p)
            assert e.value.name == "CUFSP_ERR_CUDA" and "expired" in str(e.value)
            monkeypatch.delenv("CUFSP_GRID_WAIT_NS")
        B.init(0.0, p0)
        B.advance(0.5, p)
        stats.append(B.stats)
        out.append(p.cpu().numpy())
    assert stats[0] == stats[1]
    assert np.array_equal(out[0], out[1])
