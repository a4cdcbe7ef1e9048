"""The cooperative Cholesky at the edges of its 8-column sweeps, 32- and 64-row tiles and panels,
and for pivots at the ends of the FP64 range, against NumPy's factor."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from hdsdp_b200 import _lib, api

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def _spd(n, seed):
    rng = np.random.default_rng(seed)
    G = rng.standard_normal((n, n))
    return G @ G.T / n + np.eye(n)


def _factor_and_inverse(S):
    n = S.shape[0]
    S = np.asfortranarray(S)
    L, K = np.zeros((n, n), order="F"), np.zeros((n, n), order="F")
    assert _lib.load().hdsdpb_cholesky_inverse_factor(n, api._dp(S), api._dp(L), api._dp(K)) == 0
    return L, K


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 31, 32, 33, 55, 56, 57, 63, 64, 65, 95, 96, 97, 127, 128, 129, 160,
                               191, 192, 193, 250, 320, 449, 511, 513, 700, 1025])
def test_factor_and_inverse(gpu_lib, n):
    S = _spd(n, n)
    L, K = _factor_and_inverse(S)
    ref = np.linalg.cholesky(S)
    # backward error of a Cholesky factor: at most (n + 1) eps |L||L^T| componentwise; with
    # condition number below 10 the factor and its inverse are within 20 n eps of the exact ones
    tol = 20 * max(n, 8) * EPS
    assert np.abs(L - ref).max() <= tol * np.abs(ref).max()
    assert np.abs(K @ ref - np.eye(n)).max() <= tol * 10
    assert np.array_equal(K, np.tril(K)) and np.array_equal(L, np.tril(L))


@pytest.mark.parametrize("scale", [2.0 ** -1000, 2.0 ** -520, 2.0 ** 520, 2.0 ** 1000])
@pytest.mark.parametrize("n", [5, 64, 130])
def test_pivots_of_any_size(gpu_lib, n, scale):
    """A power-of-four scale moves every pivot, exactly: the factor scales by its root."""
    S = _spd(n, 3)
    out, logdiag, ok = api.cholesky(S * scale)
    ref = np.linalg.cholesky(S) * np.sqrt(scale)
    assert ok
    assert np.abs(out - ref).max() <= 20 * max(n, 8) * EPS * np.abs(ref).max()
    assert logdiag == pytest.approx(np.log(np.diag(ref)).sum(), rel=1e-13)


def test_subnormal_and_mixed_pivots(gpu_lib):
    d = np.array([2.0 ** -1060, 1.0, 2.0 ** 900, 2.0 ** -700, 4.0, 2.0 ** -1030, 9.0, 2.0 ** 1000, 2.0 ** -2])
    out, _, ok = api.cholesky(np.diag(d))
    assert ok
    np.testing.assert_allclose(np.diag(out), np.sqrt(d), rtol=4 * EPS)


@pytest.mark.parametrize("n", [8, 64, 100, 200])
@pytest.mark.parametrize("what", ["zero", "negative", "nan", "minus_inf"])
def test_failing_pivot(gpu_lib, n, what):
    """A pivot that is not positive ends the factorisation wherever it sits."""
    for at in sorted({0, 1, 6, 7, n // 2, n - 2, n - 1}):
        S = np.eye(n) * 2.0
        S[at, at] = {"zero": 0.0, "negative": -1.0, "nan": np.nan, "minus_inf": -np.inf}[what]
        assert api.cholesky(S)[2] is False


def test_batch_is_the_grid_factor(gpu_lib):
    """One CTA a matrix and the whole-GPU kernel give the same factor to the bit."""
    lib = _lib.load()
    for n in (40, 64, 129, 250):
        S = np.stack([_spd(n, s) for s in range(3)])
        got = []
        for mode in (0, 1):
            L, K = np.zeros((3, n, n)), np.zeros((3, n, n))
            ld, st = np.zeros(3), np.zeros(3, dtype=np.int32)
            assert lib.hdsdpb_cholesky_batch(3, n, mode, api._dp(S), api._dp(L), api._dp(K), api._dp(ld),
                                             st.ctypes.data_as(C.POINTER(C.c_int))) == 0
            assert not st.any()
            got.append((L, K, ld))
        for a, b in zip(*got):
            assert np.array_equal(a, b)


def test_reciprocal_square_root_of_a_pivot(gpu_lib):
    """Diagonal matrices over the range of pivots that the straight-line reciprocal square root takes
    (2^-500 to 2^500), all mantissas and their ends: L^-1 holds it in the first column of each pair of
    columns, and in the second the square roots of the determinant and of the first pivot times it."""
    n, u = 1024, 2.0 ** -53
    rng = np.random.default_rng(0)
    edge = np.array([1.0, 1.0 + 2 * u, 1.5, 2.0 - 2 * u, 2.0, 2.0 + 4 * u, 3.0, 4.0 - 4 * u])
    sets = [rng.uniform(1.0, 4.0, n), np.tile(edge, n // edge.size), rng.uniform(1.0, 4.0, n) * 2.0 ** rng.integers(-498, 498, n),
            np.tile(edge, n // edge.size) * 2.0 ** (2 * rng.integers(-249, 249, n))]
    for d in sets:
        _, K = _factor_and_inverse(np.diag(d))
        exact = 1.0 / np.sqrt(d.astype(np.longdouble))
        err = np.abs((np.diag(K) - exact) / exact).astype(float) / u
        # 1.5 u of roundings and a margin for the iteration's own error; a second column has two of
        # these, the determinant's half rounding and two products
        assert err[0::2].max() <= 2.0
        assert err[1::2].max() <= 2 * 2.0 + 0.5 + 2.0
