"""The batched solver on one instance whose basis offsets exceed 32 bits (gpu): seven vectors of 361 million
states lie more than 2^31 doubles apart.  Against the single-instance solver with the same Krylov space: each
is within Expokit's budget delta * tol * t of the exact solution (delta = 1.2)."""
import pytest

from cuda_fsp_b200 import BatchKrylov, FSPMat, KryExpvFSP, MatrixFormat, models

pytestmark = pytest.mark.gpu


def test_offsets_beyond_32_bits(cuda):
    import torch
    m = models.mass_action((18999, 18999), [[1, 0], [-1, 0], [0, 1], [0, -1]], [[0, 0], [1, 0], [1, 0], [0, 1]],
                           [10.0, 1.0, 0.5, 0.2], name="birth_death")
    assert 6 * m.n_states > 2 ** 31
    t, tol = 0.05, 1e-8
    B = BatchKrylov.from_models([m], m=8, tol=tol)
    B.set_shape(16, 512)
    p = torch.zeros(B.total, dtype=torch.float64, device="cuda")
    grid = p.view(19000, 19000)
    grid[:3, :3] = 1.0 / 9.0
    q = p.clone()
    st = B.solve(t, p)
    assert st[0]["status"] == 0 and st[0]["t"] == t
    del B
    KryExpvFSP(t, FSPMat.from_model(m, MatrixFormat.KRONECKER), q, m=8, tol=tol, coefs=m.coefs(0)).solve()
    assert (p - q).abs().sum().item() <= 2.4 * tol * t + 1e-13
