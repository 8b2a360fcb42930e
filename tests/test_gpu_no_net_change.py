"""Reactions without net change (gpu): their gain and outflow cancel, so a network with one solves to the same
distribution, likelihood and gradient as the network without it.  A reaction whose flat shift is 0 although it
moves species leaves the box from every state and keeps its outflow."""
import numpy as np
import pytest

from cuda_fsp_b200 import FSPMat, KryExpvFSP, Likelihood, MatrixFormat, models

pytestmark = pytest.mark.gpu

BOX = (40, 60)
NU = [[1, 0], [-1, 0], [0, 1], [0, -1]]
ORDERS = [[0, 0], [1, 0], [1, 0], [0, 1]]
RATES = [10.0, 1.0, 0.5, 0.2]


def _solve(m, fmt, t=1.0, tol=1e-10):
    import torch
    v = torch.as_tensor(m.p0(), device="cuda")
    KryExpvFSP(t, FSPMat.from_model(m, getattr(MatrixFormat, fmt)), v, tol=tol, coefs=m.coefs(0)).solve()
    return v.cpu().numpy()


@pytest.mark.parametrize("fmt", ["KRONECKER", "HYB"])
def test_solution(cuda, fmt):
    plain = models.mass_action(BOX, NU, ORDERS, RATES)
    null = models.mass_action(BOX, [[0, 0]] + NU, [[1, 0]] + ORDERS, [0.3] + RATES)
    # the same table in the same order: the same solve to rounding, far below the Krylov tolerance
    assert np.abs(_solve(null, fmt) - _solve(plain, fmt)).sum() <= 1e-12


@pytest.mark.parametrize("fmt", ["KRONECKER", "HYB"])
def test_flat_shift_zero_keeps_the_outflow(cuda, fmt):
    """nu = (41, -1): every firing leaves the box.  The mass falls as exp(-0.7 t)."""
    import torch
    m = models.mass_action(BOX, [[BOX[0] + 1, -1]], [[0, 0]], [0.7])
    p = np.zeros(m.n_states)
    p[3 + (BOX[0] + 1) * 5] = 1.0
    v = torch.as_tensor(p, device="cuda")
    KryExpvFSP(1.0, FSPMat.from_model(m, getattr(MatrixFormat, fmt)), v, tol=1e-10, coefs=m.coefs(0)).solve()
    assert abs(float(v.sum()) - np.exp(-0.7)) <= 1e-9


@pytest.mark.parametrize("fmt", ["KRONECKER", "HYB"])
@pytest.mark.parametrize("nu", [4, 32768, 65536, -32768])  # flat shifts n, 2^31, 2^32 and -2^31
def test_shift_beyond_the_box_keeps_the_outflow(cuda, fmt, nu):
    import torch
    m = models.mass_action((65535, 3), [[0, nu], [1, 0]], [[0, 0], [0, 0]], [0.7, 2.0])
    p = np.zeros(m.n_states)
    p[3::65536] = 0.25
    v = torch.as_tensor(p, device="cuda")
    KryExpvFSP(1.0, FSPMat.from_model(m, getattr(MatrixFormat, fmt)), v, tol=1e-10, coefs=m.coefs(0)).solve()
    assert abs(float(v.sum()) - np.exp(-0.7)) <= 1e-9


def test_likelihood_and_gradient(cuda):
    times = np.array([0.5, 1.5])
    plain = models.mass_action(BOX, NU, ORDERS, RATES)
    null = models.mass_action(BOX, NU + [[0, 0]], ORDERS + [[1, 0]], RATES + [0.3])
    counts = np.random.default_rng(0).integers(0, 2, size=(2, BOX[1] + 1)).astype(float)
    counts[:, 12:] = 0.0
    out = [Likelihood(m, times, counts, n_marginal=1, kry_tol=1e-11).gradient() for m in (plain, null)]
    (ll0, g0), (ll1, g1) = out
    assert abs(ll1 - ll0) <= 1e-8 * abs(ll0)
    scale = np.abs(g0).max()
    assert np.abs(g1[:4] - g0).max() <= 1e-7 * scale and abs(g1[4]) <= 1e-7 * scale
