"""A call on a stream that is being captured is refused (its step control waits for the device), and what it
has queued never runs: the same object then has to work as if that call had not been made (gpu)."""
import ctypes as C
from contextlib import contextmanager

import numpy as np
import pytest

from cuda_fsp_b200 import CufspError, FSPMat, KryExpvFSP, MatrixFormat, models

pytestmark = pytest.mark.gpu


@contextmanager
def capturing(stream):
    rt = C.CDLL("libcudart.so.12")
    s = C.c_void_p(stream.cuda_stream)
    assert rt.cudaStreamBeginCapture(s, 2) == 0  # relaxed: allocations go through
    try:
        yield
    finally:
        graph = C.c_void_p()
        if rt.cudaStreamEndCapture(s, C.byref(graph)) == 0:
            rt.cudaGraphDestroy(graph)
        rt.cudaGetLastError()


@pytest.mark.parametrize("fmt", ["KRONECKER", "HYB"])
@pytest.mark.parametrize("steps_before", [0, 1, 2])
def test_krylov_solve_after_a_captured_step(cuda, fmt, steps_before):
    import torch
    m = models.toggle((90, 70))
    A = FSPMat.from_model(m, getattr(MatrixFormat, fmt))
    s = torch.cuda.Stream()
    out, stats = [], []
    for capture in (False, True):
        v = torch.as_tensor(m.p0(), device="cuda")
        torch.cuda.synchronize()
        E = KryExpvFSP(2000.0, A, v, m=20, tol=1e-9, coefs=m.coefs(0))
        for _ in range(steps_before):
            E.step(stream=s.cuda_stream)
        if capture:
            with capturing(s), pytest.raises(CufspError):
                E.step(stream=s.cuda_stream)
        stats.append(E.solve(stream=s.cuda_stream))
        out.append(v.cpu().numpy())
    assert stats[0] == stats[1] and stats[0]["n_steps"] > steps_before
    assert np.array_equal(out[0], out[1])
