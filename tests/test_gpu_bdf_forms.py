"""Which form of the BDF step a generator gets (gpu, 148 SMs): the variant of the persistent launch by states per
CTA and by terms, the basis vectors its shared memory holds, and the launch sequence where none applies."""
import re

import pytest

from cuda_fsp_b200 import BDFIntegrator, FSPMat, MatrixFormat, models

pytestmark = pytest.mark.gpu

# states per thread, near and far terms of the variant, whether the whole basis is in shared memory
FORMS = {
    "one_state": (lambda: models.toggle((210, 200), time_varying=True), "KRONECKER", 30, (1, 4, 2, True)),
    "one_state_many_far": (lambda: models.mass_action_3(bounds=(70, 20, 20)), "KRONECKER", 30, (1, 4, 8, True)),
    "two_states_many_near": (lambda: models.gene_expression((1, 1, 1, 90, 100)), "KRONECKER", 30, (2, 10, 4, True)),
    "three_states_many_far": (lambda: models.mass_action_3(bounds=(70, 50, 30)), "KRONECKER", 30, (3, 4, 8, True)),
    "one_cta": (lambda: models.toggle((12, 9), time_varying=True), "KRONECKER", 30, (1, 10, 4, True)),
    "hyb": (lambda: models.gene_expression((1, 1, 1, 40, 30)), "HYB", 30, (1, 10, 4, True)),
    "basis_partly_in_l2": (lambda: models.mass_action_3(bounds=(70, 50, 40)), "KRONECKER", 60, (3, 4, 8, False)),
    "too_many_states": (lambda: models.mass_action_3(bounds=(70, 50, 43)), "KRONECKER", 30, None),
}


@pytest.mark.parametrize("name", FORMS)
def test_form_of_the_step(cuda, name, monkeypatch):
    import torch
    make, fmt, maxl, want = FORMS[name]
    m = make()
    B = BDFIntegrator(FSPMat.from_model(m, getattr(MatrixFormat, fmt)), rtol=1e-6, atol=1e-12, maxl=maxl)
    assert B.describe() == "BDF: no step taken yet"
    p = torch.as_tensor(m.p0(), device="cuda")
    B.init(0.0, p)
    B.step(1e-3, p)
    d = B.describe()
    if want is None:
        assert d == "BDF: launch sequence"
        return
    got = re.search(r"persistent launch .* variant of (\d) states per thread, (\d+) near and (\d+) far terms, (\d+) of (\d+) basis", d)
    assert got, d
    s, near, far, slots, vecs = (int(v) for v in got.groups())
    assert (s, near, far, slots == vecs) == want, d
    assert vecs == maxl + 1


def test_new_rates_are_not_varying_rates(cuda):
    """After set_coefs no rate is added launch by launch, and the steps are those of a new integrator."""
    import numpy as np
    import torch
    m = models.gene_expression((1, 1, 1, 30, 40), time_varying=False)
    A = FSPMat.from_model(m, MatrixFormat.KRONECKER)
    c = m.coefs(0) * np.linspace(0.8, 1.2, m.nr)
    p0 = torch.as_tensor(m.p0(), device="cuda")
    out = []
    for first in (m.coefs(0), c):
        B = BDFIntegrator(A, coefs=first, rtol=1e-8, atol=1e-14)
        p = p0.clone()
        if first is not c:
            B.init(0.0, p0)
            B.advance(0.5, p)
            B.set_coefs(c)
        B.init(0.0, p0)
        B.advance(1.0, p)
        assert " 0 rates added" in B.describe()
        out.append((p.cpu().numpy(), B.stats))
    assert out[0][1] == out[1][1]
    assert np.array_equal(out[0][0], out[1][0])


def test_varying_rates_are_counted(cuda):
    import torch
    m = models.gene_expression((1, 1, 1, 30, 40))  # one switching rate
    B = BDFIntegrator(FSPMat.from_model(m, MatrixFormat.KRONECKER), rtol=1e-6, atol=1e-12)
    p = torch.as_tensor(m.p0(), device="cuda")
    B.init(0.0, p)
    B.advance(1.0, p)
    assert " 1 rates added" in B.describe()


def _advance():
    import torch
    m = models.gene_expression((1, 1, 1, 30, 40))
    B = BDFIntegrator(FSPMat.from_model(m, MatrixFormat.KRONECKER), rtol=1e-8, atol=1e-14)
    p = torch.as_tensor(m.p0(), device="cuda")
    B.init(0.0, p)
    B.advance(1.0, p)
    return p.cpu().numpy(), B.describe()


def test_report_copied_instead_of_polled(cuda, tmp_path):
    """CUFSP_BDF_SPIN=0 holds for the persistent step, too."""
    import os
    import subprocess
    import sys
    from pathlib import Path

    import numpy as np
    root = Path(__file__).resolve().parent.parent
    code = ("import sys; sys.path[:0] = [%r, %r]\nimport numpy as np, test_gpu_bdf_forms as t\np, d = t._advance()\n"
            "assert d.endswith('report copied'), d\nnp.save(%r, p)" % (str(root), str(root / "tests"), str(tmp_path / "p.npy")))
    subprocess.run([sys.executable, "-c", code], check=True, env={**os.environ, "CUFSP_BDF_SPIN": "0"})
    p, d = _advance()
    assert d.endswith("report polled"), d
    assert np.array_equal(np.load(tmp_path / "p.npy"), p)
