"""Cholesky factorisations that meet a pivot that is not positive, as a line search's trial points
do all the time: the answer is "not positive definite", never an error, and what is factored
beside them is unharmed."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from hdsdp_b200 import _lib, api, instances

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps
DENSE_SDP = 4   # cone_type, interface/hdsdp_conic.h


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


@pytest.mark.parametrize("n,fused", [(500, True), (1000, True), (2000, True), (1000, False), (2100, False), (2500, True),
                                     (4200, True), (3700, False)])
def test_blocks(gpu_lib, n, fused):
    """One launch (with and without K) and the recursive forms (with K above 2048 rows, without
    above 3584): a failure in the first, a middle and the last diagonal block, and last the good
    matrix on the memory that they leave behind."""
    lib = _lib.load()
    rng = np.random.default_rng(n)
    G = rng.standard_normal((n, 40))
    good = G @ G.T / 40.0 + np.eye(n)
    L, K = np.zeros((n, n), order="F"), np.zeros((n, n), order="F")

    def factor(S):
        if fused:
            return lib.hdsdpb_cholesky_inverse_factor(n, api._dp(S), api._dp(L), api._dp(K))
        return lib.hdsdpb_cholesky(n, api._dp(S), api._dp(L), None)

    for at in (3, 63, 64, 64 * (n // 128) + 17, 64 * ((n - 1) // 64), n - 1):
        S = good.copy()
        S[at, at] = -1.0    # a diagonal entry below zero fails its pivot, whatever the rest
        assert factor(S) == 1
    assert factor(good) == 0
    # backward error of the factor: at most (n + 1) eps |L||L^T| componentwise
    r = np.abs(np.tril(L) @ (np.tril(L).T @ np.ones(n)) - good @ np.ones(n))
    assert (r <= 4 * n * EPS * (np.abs(L) @ (np.abs(L).T @ np.ones(n)))).all()
    if fused:
        x = rng.standard_normal(n)
        # |L K - I| <= c n eps |L||K||L||K| componentwise, block by block
        aL, aK = np.abs(L), np.abs(K)
        assert (np.abs(L @ (K @ x) - x) <= 8 * n * EPS * (aL @ (aK @ (aL @ (aK @ np.abs(x)))))).all()


@pytest.mark.parametrize("n", [40, 130, 700, 2100])
def test_line_search_on_one_cone(gpu_lib, n):
    """Trial points of one cone, inside and outside in turn: the log barrier of an inside point is
    the same to the bit whatever was refused before it."""
    lib = _lib.load()
    inst = instances.maxcut(n, seed=n, n_edges=4 * n, weights=(0.5, 1.5))
    rows, vals = inst.column(0)
    start = instances.pack_idx(n, np.arange(n), np.arange(n))
    at = np.searchsorted(rows, start)
    diag = np.where(rows[np.minimum(at, rows.size - 1)] == start, vals[np.minimum(at, rows.size - 1)], 0.0)
    y = 2.0 * diag - 1.0    # S = C - diag(y) is diagonally dominant
    keep = [np.ascontiguousarray(inst.Ap, np.int32), np.ascontiguousarray(inst.Ai, np.int32), np.ascontiguousarray(inst.Ax)]
    user, cone, inside, value = C.c_void_p(), C.c_void_p(), C.c_int(), C.c_double()
    ip = C.POINTER(C.c_int)
    assert lib.HUserDataCreate(C.byref(user)) == 0
    lib.HUserDataSetConeData(user, DENSE_SDP, n, n, keep[0].ctypes.data_as(ip), keep[1].ctypes.data_as(ip), api._dp(keep[2]))
    assert lib.HConeCreate(C.byref(cone)) == 0 and lib.HConeSetData(cone, user) == 0
    assert lib.HConeProcData(cone) == 0 and lib.HConePresolveData(cone) == 0
    lib.HConeSetStart(cone, 0.0)
    try:
        seen = []
        for where in (None, 0, None, n // 2, n - 1, None):
            t = y.copy()
            if where is not None:
                t[where] += 50.0
            assert lib.HConeCheckIsInterior(cone, 1.0, api._dp(t), C.byref(inside)) == 0
            assert inside.value == (where is None)
            if where is None:
                assert lib.HConeGetLogBarrier(cone, 0.0, None, 0, C.byref(value)) == 0
                seen.append(value.value)
        assert seen[0] == seen[1] == seen[2]
    finally:
        lib.HConeDestroy(C.byref(cone))
        lib.HUserDataDestroy(C.byref(user))
