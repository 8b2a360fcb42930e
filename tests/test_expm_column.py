"""The first column of the exponential of an upper Hessenberg matrix, which the Krylov step control takes
(cufsp::expm_hessenberg_col), against the full Pade exponential and SciPy's: sizes around the padding to 8,
norms on both sides of the direct and the squaring form.  The matrices are generator-like (columns sum to
at most 0 before the augmentation), so that exp does not grow and rounding moves the column by a small
multiple of u * max(1, norm)."""
import ctypes as C

import numpy as np
import pytest
import scipy.linalg

from cuda_fsp_b200 import CufspError, expm


def column(built, a):
    lib = C.CDLL(str(built["libcufsp"]))
    f = lib._ZN5cufsp19expm_hessenberg_colEiPKdPd
    A = np.asfortranarray(a, dtype=np.float64)
    out = np.empty(A.shape[0])
    dp = lambda v: v.ctypes.data_as(C.POINTER(C.c_double))  # noqa: E731
    return f(A.shape[0], dp(A), dp(out)), out


@pytest.mark.parametrize("k", [1, 2, 7, 8, 9, 17, 32, 33, 62])
@pytest.mark.parametrize("norm", [0.0, 0.3, 5.0, 20.0, 43.0, 60.0, 700.0])
def test_column_matches_full_exponential(built, k, norm):
    rng = np.random.default_rng(k)
    h = np.triu(np.abs(rng.normal(size=(k, k))), -1)
    h -= np.diag(h.sum(axis=0) + np.diag(h))
    s = np.abs(h).sum(axis=0).max()
    a = h * (norm / s if s > 0 else 0.0)
    rc, col = column(built, a)
    assert rc == 0
    bar = 64 * 2.0 ** -53 * max(1.0, norm)
    assert np.linalg.norm(col - expm(a)[:, 0]) <= bar
    assert np.linalg.norm(col - scipy.linalg.expm(a)[:, 0]) <= bar


def test_column_reports_nonfinite(built):
    a = np.triu(np.ones((5, 5)), -1)
    a[1, 2] = np.nan
    assert column(built, a)[0] == 5  # CUFSP_ERR_NONFINITE
    with pytest.raises(CufspError):
        expm(a)
