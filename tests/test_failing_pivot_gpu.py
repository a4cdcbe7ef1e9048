"""Cholesky factorisations that meet a pivot that is not positive, as a line search's trial points
do all the time: the answer is "not positive definite", never an error, and what is factored
beside them is unharmed."""
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


def _failing(S, at):
    """S with its pivot `at` made -1; the pivots before it stay as they are."""
    S = S.copy()
    L = np.linalg.cholesky(S)
    S[at, at] -= L[at, at] ** 2 + 1.0
    return S


@pytest.mark.parametrize("mode", [0, 1], ids=["one_cta", "grid"])
@pytest.mark.parametrize("n", [64, 200])
def test_every_sweep(gpu_lib, n, mode):
    """A failure in each 8-column sweep of each diagonal block, first and last column of it, with a
    good matrix behind each bad one."""
    good = _spd(n, n)
    ref = np.linalg.cholesky(good)
    at = sorted({a for s in range(0, n, 8) for a in (s, min(s + 7, n - 1))})
    S = np.stack([M for a in at for M in (_failing(good, a), good)])
    count = len(S)
    L, K = np.zeros((count, n, n)), np.zeros((count, n, n))
    ld, st = np.zeros(count), np.zeros(count, dtype=np.int32)
    assert _lib.load().hdsdpb_cholesky_batch(count, n, mode, api._dp(S), api._dp(L), api._dp(K), api._dp(ld),
                                             st.ctypes.data_as(C.POINTER(C.c_int))) == 0
    assert st.tolist() == [1, 0] * len(at)
    # condition number below 10: the factor and its inverse are within 20 n eps of the exact ones
    for q in range(1, count, 2):
        assert np.abs(L[q].T - ref).max() <= 20 * n * EPS * np.abs(ref).max()
        assert np.abs(K[q].T @ ref - np.eye(n)).max() <= 200 * n * EPS
