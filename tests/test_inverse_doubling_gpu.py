"""The inverse of a factor whose factorisation does not form it, at orders where the doubling's last
pair is one row, one whole block, or missing at some levels, against the matrix itself."""
import ctypes as C

import numpy as np
import pytest

from hdsdp_b200 import _lib, api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2049, 2111, 2112, 2113, 2176, 2177, 2305, 3073])
def test_inverse_by_doubling(n):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) / np.sqrt(n)
    S = A @ A.T + np.eye(n)          # eigenvalues in about [1, 5]
    X = np.empty((n, n))
    assert _lib.load().hdsdpb_inverse(n, api._dp(S), api._dp(X)) == 0
    # |S X - I| <= c n eps |S| |X| for a backward stable factor and triangular inverse; the 2-norms
    # are at most 6 and 1, and 8 covers the three n^3 stages
    assert np.abs(S @ X - np.eye(n)).max() <= 8 * n * np.finfo(float).eps * 6
    assert np.array_equal(X, X.T)
