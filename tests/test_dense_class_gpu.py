"""The dense-coefficient class (all matrices in shared launches) against the NumPy restatement:
orders and counts around the 64-wide tiles and the scratch chunk (32 matrices at order 1000),
alone and mixed with sparse and rank-one coefficients. Bar: 1e-11 relative, the bar of the Schur
parity tests."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from hdsdp_b200 import _lib, api, instances
from oracle import kernels_ref as K

pytestmark = pytest.mark.gpu


def _problem(n, m, mixed, seed):
    rng = np.random.default_rng(seed)
    mats = [np.eye(n) + 0.1 * np.diag(rng.uniform(-1, 1, n))]
    for t in range(m):
        A = np.zeros((n, n))
        if mixed and t % 3 == 1:
            A[t % n, t % n] = 1.0
        elif mixed and t % 3 == 2:
            i, j = (t * 7) % n, (t * 11 + 1) % n
            A[i, j] = A[j, i] = 0.5
        else:
            R = rng.standard_normal((n, n))
            A = (R + R.T) / 2.0
        mats.append(A)
    return instances._assemble("dense_class", n, instances._dense_columns(n, mats), np.zeros(m)), mats


@pytest.mark.parametrize("n,m,mixed", [(4, 1, False), (33, 7, False), (64, 64, False), (65, 65, False),
                                       (80, 130, False), (40, 31, True), (97, 20, True), (1000, 33, False)])
def test_dense_class(gpu_lib, n, m, mixed):
    inst, mats = _problem(n, m, mixed, n + m)
    rng = np.random.default_rng(1)
    y = rng.uniform(-1, 1, m) * 0.1 / np.sqrt(n * m)
    resi = -0.5
    r = api.schur_probe(inst, y, resi)
    C, A = mats[0], np.stack(mats[1:])
    W = np.linalg.inv(C - np.einsum("k,kij->ij", y, A) - resi * np.eye(n))
    WA = (W @ A).reshape(m, -1)
    M = np.tril(WA @ (A @ W).reshape(m, -1).T)   # tr(W A_i W A_j)
    flat = A.reshape(m, -1)
    for got, want in ((r["M"], M), (r["asinv"], flat @ W.ravel()), (r["asinvrd"], resi * (flat @ (W @ W).ravel()))):
        assert np.abs(got - want).max() <= 1e-11 * max(1.0, np.abs(want).max())


def test_dense_class_primal_dual(gpu_lib):
    """The slack is assembled from every matrix of the class (log det S against NumPy's)."""
    inst, mats = _problem(70, 25, True, 3)
    y = np.random.default_rng(2).uniform(-1, 1, 25) * 0.002
    _, logdet = api.ratio_probe(inst, y, 0.0, 0.1 * y, 0.0)
    S = K.dual_slack(mats[0], mats[1:], y)
    assert logdet == pytest.approx(np.linalg.slogdet(S)[1], rel=1e-12, abs=1e-11)


def test_more_matrices_than_a_grid_has_rows(gpu_lib):
    """<A_i, X> over 65,537 dense 3 x 3 matrices of one cone, whose scratch stays in proportion: below
    2 GB (a set of 256 MB for each product and each part of their inner products), where every pair of
    matrices would take 34 GB."""
    import torch

    n, m = 3, 65537
    rng = np.random.default_rng(4)
    R = rng.standard_normal((m + 1, n, n))
    A = (R + R.transpose(0, 2, 1)) / 2.0
    c, r = np.triu_indices(n)   # column by column of the lower triangle
    pos = instances.pack_idx(n, r, c)
    Ap = np.ascontiguousarray(pos.size * np.arange(m + 2), np.int32)
    Ai = np.ascontiguousarray(np.tile(pos, m + 1), np.int32)
    Ax = np.ascontiguousarray(A[:, r, c]).ravel()
    X = R[0] @ R[0].T
    L, ip = _lib.load(), C.POINTER(C.c_int)
    user, cone, out = C.c_void_p(), C.c_void_p(), np.zeros(m)
    assert L.HUserDataCreate(C.byref(user)) == 0
    L.HUserDataSetConeData(user, 4, m, n, Ap.ctypes.data_as(ip), Ai.ctypes.data_as(ip), api._dp(Ax))
    assert L.HConeCreate(C.byref(cone)) == 0 and L.HConeSetData(cone, user) == 0
    L.hdsdpb_release_cached_memory()
    before = torch.cuda.mem_get_info()[0]
    try:
        assert L.HConeProcData(cone) == 0 and L.HConePresolveData(cone) == 0
        L.HConeComputeATimesX(cone, api._dp(X), api._dp(out))
        assert before - torch.cuda.mem_get_info()[0] < 2 << 30
    finally:
        L.HConeDestroy(C.byref(cone))
        L.HUserDataDestroy(C.byref(user))
        L.hdsdpb_release_cached_memory()
    want = np.einsum("kij,ij->k", A[1:], X)
    assert np.abs(out - want).max() <= 1e-11 * np.abs(want).max()
