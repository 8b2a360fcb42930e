"""Batched gradients above the size up to which the workers share the SMs: every worker's persistent pass
takes the whole GPU, as a single call's does, so both do the same arithmetic in the same order."""
import numpy as np
import pytest

from cuda_fsp_b200 import Likelihood, generate_data, histograms, models

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [113, 127])  # 103,968 states, just past 148 x 700, and 131,072
def test_turns_equal_single_calls(cuda, monkeypatch, side):
    monkeypatch.delenv("CUFSP_GRAD_SM_SHARE", raising=False)
    m = models.gene_expression((1, 1, 1, side, side), time_varying=False)
    times = np.array([1.0, 4.0])
    counts, outside = histograms(generate_data(m, times, [0, 0, 0, 0, 0], 200, seed=11), m.bounds, n_marginal=3)
    L = Likelihood(m, times, counts, outside=outside, n_marginal=3, kry_tol=1e-8)
    rng = np.random.default_rng(3)
    sets = np.stack([m.coefs(0) * 10.0 ** rng.uniform(-0.3, 0.3, m.nr) for _ in range(3)])
    ll_b, g_b = L.gradient_batched(sets, workers=4)
    for i in range(len(sets)):
        ll, g = L.gradient(sets[i])
        assert abs(ll_b[i] - ll) <= 1e-13 * abs(ll)
        assert np.abs(g_b[i] - g).max() <= 1e-12 * np.abs(g).max()
