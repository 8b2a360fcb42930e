"""The persistent Arnoldi pass at the edges of its variants (gpu): one, two and four states per thread,
few and many near and far shifts, the general variant whose slices leave only part of the basis in
shared memory, windows of incomplete orthogonalisation that fit shared memory or do not, one CTA and a
last CTA with a partial slice.  Against the oracle's Krylov solve of the same tolerance: each is within
Expokit's global budget delta * tol * t of the exact solution (delta = 1.2), so they differ by at most
twice that."""
import numpy as np
import pytest

import oracle
from cuda_fsp_b200 import FSPMat, KryExpvFSP, MatrixFormat, models

pytestmark = pytest.mark.gpu


def _bd(b0, b1):
    return models.mass_action((b0, b1), [[1, 0], [-1, 0], [0, 1], [0, -1]], [[0, 0], [1, 0], [1, 0], [0, 1]],
                              [10.0, 1.0, 0.5, 0.2], name="birth_death")


CASES = {
    "one_cta": (lambda: models.toggle((12, 9)), "KRONECKER", 5.0, dict(m=20)),
    "one_state_last_partial": (lambda: _bd(130, 247), "KRONECKER", 1.0, dict(m=30)),
    "two_states": (lambda: models.toggle((210, 200)), "KRONECKER", 20.0, dict(m=25)),
    "four_states": (lambda: _bd(300, 300), "KRONECKER", 0.5, dict(m=30)),
    "many_near_terms": (lambda: models.gene_expression((1, 1, 1, 90, 60), time_varying=False), "KRONECKER", 1.0, dict(m=30)),
    "many_far_terms": (lambda: models.mass_action_3(bounds=(70, 20, 20)), "KRONECKER", 0.05, dict(m=30)),
    "basis_partly_in_l2": (lambda: models.mass_action_3(bounds=(70, 60, 40)), "KRONECKER", 0.01, dict(m=30)),
    "basis_partly_in_l2_hyb": (lambda: models.mass_action_3(bounds=(70, 60, 40)), "HYB", 0.01, dict(m=30)),
    "window_in_slots": (lambda: _bd(160, 240), "KRONECKER", 0.5, dict(m=30, iop=True, q_iop=3)),
    "window_of_one": (lambda: _bd(60, 90), "KRONECKER", 0.1, dict(m=20, iop=True, q_iop=1)),
    "window_beyond_slots": (lambda: models.mass_action_3(bounds=(70, 60, 40)), "KRONECKER", 0.01,
                            dict(m=30, iop=True, q_iop=26)),
    "largest_m": (lambda: _bd(130, 90), "KRONECKER", 2.0, dict(m=60)),
    "smallest_m": (lambda: _bd(40, 60), "KRONECKER", 1e-8, dict(m=1)),
}


@pytest.mark.parametrize("name", CASES)
def test_persistent_pass_variants(cuda, name):
    import torch
    make, fmt, t, kw = CASES[name]
    m, tol = make(), 1e-9
    p = np.random.default_rng(3).uniform(0.0, 1.0, m.n_states)
    # mass away from the upper faces, smooth enough that a few steps reach t
    x = np.stack(np.unravel_index(np.arange(m.n_states), [b + 1 for b in reversed(m.bounds)]))[::-1]
    p *= np.exp(-0.5 * sum(x[s] / (1.0 + 0.2 * b) for s, b in enumerate(m.bounds)))
    p /= p.sum()
    A = FSPMat.from_model(m, getattr(MatrixFormat, fmt))
    v = torch.as_tensor(p, device="cuda")
    st = KryExpvFSP(t, A, v, tol=tol, coefs=m.coefs(0), **kw).solve()
    assert st["t_now"] == t
    w, _, rc = oracle.expv(oracle.assemble_model(m), m.coefs(0), t, p, tol=tol, **kw)
    assert rc == 0
    assert np.abs(v.cpu().numpy() - w).sum() <= 2.4 * tol * max(t, 1.0)
