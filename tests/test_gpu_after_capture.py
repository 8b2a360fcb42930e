"""A call on a stream that is being captured is refused (its step control waits for the device), and what it
has queued never runs: the same object then has to work as if that call had not been made (gpu)."""
import ctypes as C
from contextlib import contextmanager

import numpy as np
import pytest

from cuda_fsp_b200 import BDFIntegrator, CufspError, FSPMat, KryExpvFSP, MatrixFormat, models

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


@pytest.mark.parametrize("steps_before", [0, 1, 4])
def test_bdf_after_a_captured_step(cuda, steps_before):
    """The captured attempt is the first with new rates, so that it has rebuilt the coefficient table (given an
    initial step, the start of an integration waits for nothing)."""
    import torch
    m = models.toggle((50, 41))
    c = m.coefs(0) * np.linspace(0.7, 1.3, m.nr)
    s = torch.cuda.Stream()
    out, stats = [], []
    for capture in (False, True):
        A = FSPMat.from_model(m, MatrixFormat.HYB)
        p0 = torch.as_tensor(m.p0(), device="cuda")
        p = p0.clone()
        torch.cuda.synchronize()
        B = BDFIntegrator(A, coefs=m.coefs(0), rtol=1e-8, atol=1e-14, h_init=1e-3)
        B.init(0.0, p0, stream=s.cuda_stream)
        for _ in range(steps_before):
            B.step(50.0, p, stream=s.cuda_stream)
        B.set_coefs(c)
        if capture:
            with capturing(s):
                B.init(0.0, p0, stream=s.cuda_stream)
                with pytest.raises(CufspError):
                    B.advance(50.0, p, stream=s.cuda_stream)
        B.init(0.0, p0, stream=s.cuda_stream)
        B.advance(50.0, p, stream=s.cuda_stream)
        stats.append(B.stats)
        out.append(p.cpu().numpy())
    assert stats[0] == stats[1]
    assert np.array_equal(out[0], out[1])
