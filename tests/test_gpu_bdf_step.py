"""The BDF step attempt as one persistent launch at the edges of its variants (gpu): one, two and three
states per thread, few and many near and far shifts, rates that vary and rates that do not, a GMRES space
too small to converge (the step is halved), more basis vectors than shared memory holds, the sparse
format.  Against the oracle's BDF with the same tolerances: the two make the same decisions up to
rounding, and either stays within 100 rtol of the exact solution in 1-norm on these horizons."""
import numpy as np
import pytest

import oracle
from cuda_fsp_b200 import BDFIntegrator, FSPMat, MatrixFormat, models

pytestmark = pytest.mark.gpu

CASES = {
    "one_state": (lambda: models.toggle((210, 200), time_varying=True), "KRONECKER", [30.0, 100.0], {}),
    "one_state_many_far": (lambda: models.mass_action_3(bounds=(70, 20, 20)), "KRONECKER", [0.01], {}),
    "two_states_many_near": (lambda: models.gene_expression((1, 1, 1, 90, 100)), "KRONECKER", [0.5, 1.0], {}),
    "three_states_many_far": (lambda: models.mass_action_3(bounds=(70, 50, 30)), "KRONECKER", [0.002], {}),
    "one_cta": (lambda: models.toggle((12, 9), time_varying=True), "KRONECKER", [100.0], {}),
    "hyb": (lambda: models.gene_expression((1, 1, 1, 40, 30)), "HYB", [1.0], {}),
    "small_krylov_space": (lambda: models.toggle((31, 31), time_varying=True), "KRONECKER", [200.0], dict(maxl=1)),
    "basis_partly_in_l2": (lambda: models.mass_action_3(bounds=(70, 50, 40)), "KRONECKER", [0.02],
                           dict(maxl=60, eps_lin=1e-12, rtol=1e-6)),
    "largest_krylov_space": (lambda: models.gene_expression((1, 1, 1, 20, 30)), "KRONECKER", [2.0], dict(maxl=60)),
}


@pytest.mark.parametrize("name", CASES)
def test_bdf_step_variants(cuda, name):
    import torch
    make, fmt, times, kw = CASES[name]
    m, kw = make(), {"rtol": 1e-9, "atol": 1e-14, **kw}
    A = FSPMat.from_model(m, getattr(MatrixFormat, fmt))
    B = BDFIntegrator(A, **kw)
    p = torch.as_tensor(m.p0(), device="cuda")
    B.init(0.0, p)
    ref, rst, rc = oracle.bdf(oracle.assemble_model(m), m.coefs, 0.0, m.p0(), times, **kw)
    assert rc == 0
    for k, t in enumerate(times):
        assert B.advance(t, p) == t
        assert np.abs(p.cpu().numpy() - ref[k]).sum() <= 100 * kw["rtol"]
    st = B.stats
    assert abs(st["n_steps"] - rst["n_steps"]) <= max(3, rst["n_steps"] // 20), (st, rst)
    assert (st["n_lin_fail"] > 0) == (rst["n_lin_fail"] > 0)
