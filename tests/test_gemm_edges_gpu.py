"""GEMM at the edges of its tiles: ends of M, N and K in every position, 16-byte and element-wise
copies (even and odd leading dimensions), both tile sizes, against NumPy in float64."""
import ctypes as C

import numpy as np
import pytest

from hdsdp_b200 import _lib

pytestmark = pytest.mark.gpu


def _ptr(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


def _padded(rng, rows, cols, ld):
    """A column-major rows x cols matrix whose padding holds NaN."""
    buf = np.full((cols, ld), np.nan)
    buf[:, :rows] = rng.standard_normal((cols, rows))
    return buf, buf[:, :rows].T


@pytest.mark.parametrize("ta", [0, 1])
@pytest.mark.parametrize("tb", [0, 1])
@pytest.mark.parametrize("m,n,k,pad", [
    (1, 1, 1, 1), (1, 33, 16, 0), (33, 1, 17, 1), (31, 32, 15, 0), (32, 31, 16, 1), (65, 33, 96, 0),
    (63, 64, 81, 1), (64, 66, 80, 2), (127, 65, 3, 0), (200, 201, 79, 0), (130, 130, 0, 0),
    (3073, 3073, 35, 0), (3072, 3073, 48, 1),
])
def test_gemm_edges(m, n, k, pad, ta, tb):
    lib = _lib.load()
    rng = np.random.default_rng(m * 7 + n * 3 + k)
    ar, ac, br, bc = (k, m, n, k) if ta and tb else (k, m, k, n) if ta else (m, k, n, k) if tb else (m, k, k, n)
    lda, ldb, ldc = max(1, ar) + pad, max(1, br) + pad, m + pad
    if pad != 1:   # even leading dimensions
        lda, ldb = lda + lda % 2, ldb + ldb % 2
    abuf, a = _padded(rng, ar, ac, lda)
    bbuf, b = _padded(rng, br, bc, ldb)
    cbuf, c = _padded(rng, m, n, ldc)
    opa, opb = (a.T if ta else a), (b.T if tb else b)
    want = 0.75 * (opa @ opb) - 0.5 * c
    # each of the two sums over k carries at most k roundings of the products' magnitudes
    bound = 4 * (k + 4) * 2.0 ** -53 * (0.75 * (np.abs(opa) @ np.abs(opb)) + 0.5 * np.abs(c))
    lib.hdsdpb_gemm.argtypes = [C.c_int] * 3 + [C.c_double, C.POINTER(C.c_double), C.c_int, C.c_int, C.POINTER(C.c_double),
                                                C.c_int, C.c_int, C.c_double, C.POINTER(C.c_double), C.c_int]
    assert lib.hdsdpb_gemm(m, n, k, 0.75, _ptr(abuf), lda, ta, _ptr(bbuf), ldb, tb, -0.5, _ptr(cbuf), ldc) == 0
    assert (np.abs(c - want) <= bound).all()
    assert np.isnan(cbuf[:, m:]).all()


@pytest.mark.parametrize("tb", [0, 1])
def test_more_column_tiles_than_a_grid_has(tb):
    """65,535 tiles of 32 columns and one more column, which takes a second launch."""
    lib = _lib.load()
    m, n, k = 3, 65535 * 32 + 1, 2
    rng = np.random.default_rng(tb)
    a = np.asfortranarray(rng.standard_normal((m, k)))
    b = rng.standard_normal((n, k)) if tb else rng.standard_normal((k, n))
    b = np.asfortranarray(b)
    c = np.zeros((m, n), order="F")
    lib.hdsdpb_gemm.argtypes = [C.c_int] * 3 + [C.c_double, C.POINTER(C.c_double), C.c_int, C.c_int, C.POINTER(C.c_double),
                                                C.c_int, C.c_int, C.c_double, C.POINTER(C.c_double), C.c_int]
    assert lib.hdsdpb_gemm(m, n, k, 1.0, _ptr(a), m, 0, _ptr(b), n if tb else k, tb, 0.0, _ptr(c), m) == 0
    op = b.T if tb else b
    assert (np.abs(c - a @ op) <= 4 * (k + 4) * 2.0 ** -53 * (np.abs(a) @ np.abs(op))).all()
