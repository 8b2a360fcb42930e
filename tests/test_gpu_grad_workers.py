"""Batched gradients with so many workers that a share of the SMs cannot hold the generator's slices, and Krylov
solves of generators that the whole GPU cannot (gpu): both take another path, with the same results."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from cuda_fsp_b200 import FSPMat, KryExpvFSP, Likelihood, MatrixFormat, generate_data, histograms, models

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent


@pytest.mark.parametrize("share", [None, "1"])
@pytest.mark.parametrize("workers,side", [(32, 89), (24, 107)])  # 64,800 states on 4 CTAs, 93,312 on 6
def test_many_workers(cuda, monkeypatch, workers, side, share):
    if share is None:
        monkeypatch.delenv("CUFSP_GRAD_SM_SHARE", raising=False)
    else:
        monkeypatch.setenv("CUFSP_GRAD_SM_SHARE", share)
    m = models.gene_expression((1, 1, 1, side, side), time_varying=False)
    times = np.array([0.5, 1.0])
    counts, outside = histograms(generate_data(m, times, [0, 0, 0, 0, 0], 200, seed=11), m.bounds, n_marginal=3)
    L = Likelihood(m, times, counts, outside=outside, n_marginal=3, kry_tol=1e-8)
    rng = np.random.default_rng(3)
    sets = np.stack([m.coefs(0) * 10.0 ** rng.uniform(-0.3, 0.3, m.nr) for _ in range(workers)])
    ll_b, g_b = L.gradient_batched(sets, workers=workers)
    for i in (0, workers // 2, workers - 1):  # whole-GPU passes in turn: the single call's arithmetic
        ll, g = L.gradient(sets[i])
        assert abs(ll_b[i] - ll) <= 1e-13 * abs(ll)
        assert np.abs(g_b[i] - g).max() <= 1e-12 * np.abs(g).max()


def _solve():
    import torch
    m = models.mass_action_3(bounds=(131, 130, 129))  # 2,247,960 states: 15,190 per CTA
    v = torch.as_tensor(m.p0(), device="cuda")
    KryExpvFSP(1e-3, FSPMat.from_model(m, MatrixFormat.KRONECKER), v, m=10, tol=1e-8, coefs=m.coefs(0)).solve()
    return v.cpu().numpy()


def test_size_limit_raised_beyond_what_fits(cuda, tmp_path):
    code = ("import sys; sys.path[:0] = [%r, %r]\nimport numpy as np, test_gpu_grad_workers as t\nnp.save(%r, t._solve())"
            % (str(ROOT), str(ROOT / "tests"), str(tmp_path / "v.npy")))
    subprocess.run([sys.executable, "-c", code], check=True, env={**os.environ, "CUFSP_ARNOLDI_MAX_N": str(1 << 22)})
    assert np.array_equal(np.load(tmp_path / "v.npy"), _solve())  # the launch sequence in both
