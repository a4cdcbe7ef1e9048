"""Solves with a recursively factored matrix: two, three and more diagonal blocks, the last one odd."""
import ctypes as C

import numpy as np
import pytest

from hdsdp_b200 import _lib, api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3584, 3585, 4097, 5151, 6500])
def test_recursive_solve(n):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) / np.sqrt(n)
    S = A @ A.T + 0.1 * np.eye(n)
    b = rng.standard_normal(n)
    x = np.empty(n)
    assert _lib.load().hdsdpb_cholesky_solve(n, api._dp(S), api._dp(b), api._dp(x)) == 0
    # normwise backward error of a Cholesky solve: |b - S x| <= c n eps |S| |x|, |S|_2 <= 4.2
    assert np.linalg.norm(b - S @ x) <= 4 * n * np.finfo(float).eps * 4.2 * np.linalg.norm(x)


@pytest.mark.parametrize("n", [200, 3585, 5151])
def test_solve_with_a_copied_factor(n):
    """A factor copied over one of another matrix solves with its own blocks."""
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) / np.sqrt(n)
    S = A @ A.T + 0.1 * np.eye(n)
    S0 = S + np.diag(rng.uniform(0.5, 2.0, n))
    b = rng.standard_normal(n)
    x = np.empty(n)
    assert _lib.load().hdsdpb_cholesky_copy_solve(n, api._dp(S0), api._dp(S), api._dp(b), api._dp(x)) == 0
    # as above: |b - S x| <= c n eps |S| |x|, |S|_2 <= 4.2
    assert np.linalg.norm(b - S @ x) <= 4 * n * np.finfo(float).eps * 4.2 * np.linalg.norm(x)
