"""The batched solver on vectors that start on an 8-byte boundary only (gpu): a view into a larger buffer
gives the bits of the aligned solve, leaves what lies around it alone, and the two alternate on one solver."""
import numpy as np
import pytest

from cuda_fsp_b200 import BatchKrylov, models

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 128), (8, 256), (0, 0)])  # (0, 0): the autotuner's first solve
def test_view_gives_the_aligned_result(cuda, shape, monkeypatch, tmp_path):
    import torch
    monkeypatch.setenv("CUFSP_AUTOTUNE_CACHE", str(tmp_path / "tune.txt"))
    ms = [models.toggle(b) for b in [(30, 21), (6, 4), (40, 40), (2, 2)]] * 3  # odd and even sizes
    B = BatchKrylov.from_models(ms, m=20, tol=1e-9)
    if shape != (0, 0):
        B.set_shape(*shape)
    p0 = B.pack([mm.p0() for mm in ms])
    buf = torch.full((B.total + 2,), 7.0, dtype=torch.float64, device="cuda")
    view = buf[1:1 + B.total]
    assert p0.data_ptr() % 16 == 0 and view.data_ptr() % 16 == 8
    view.copy_(p0)
    st_view = B.solve(50.0, view)
    p = p0.clone()
    st = B.solve(50.0, p)
    assert st_view == st
    assert np.array_equal(view.cpu().numpy(), p.cpu().numpy())
    assert buf[0].item() == 7.0 and buf[-1].item() == 7.0
    view.copy_(p0)
    B.solve(50.0, view)
    assert np.array_equal(view.cpu().numpy(), p.cpu().numpy())
