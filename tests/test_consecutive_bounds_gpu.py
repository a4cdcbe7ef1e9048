"""Step bounds taken one after the other on one cone: what lives from one to the next (the warm start
vector, how many steps the last one took, the exchange words and their tags, the lists of the step
matrix's entries) against a NumPy restatement of the reference's estimator that is started the same
way (linalg/hdsdp_lanczos.c:33-53, :161-292): the perturbed image of the last Ritz vector, whose sign
an eigensolver leaves open. One order for each kernel. Bar: 1e-8 relative, that of the step parity
tests."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from hdsdp_b200 import _lib, api, instances
from test_grid_lanczos_gpu import _direction

pytestmark = pytest.mark.gpu

DENSE_SDP, VAR = 4, 0   # cone_type and buffer, interface/hdsdp_conic.h
KINDS = ["dense", "diag", "hub", "band64", "spike"]
# a direction with one eigenvalue far out takes few steps, most others many
ORDER = ["dense", "dense", "spike", "spike", "diag", "hub", "spike", "band64", "band64", "dense", "hub", "diag"]


def _raw_vector(n):
    libc = C.CDLL(None)
    libc.srand(n)
    v = np.zeros(n)
    for i in range(n):
        libc.srand(libc.rand())
        r1, r2 = libc.rand() % 1627, libc.rand() % 2
        v[i] = np.sqrt(np.sqrt(float(r1))) * (r2 - 0.5)
    return v


def _bound(op, start, maxdim=30):
    """The estimator's step bound from a start vector, the image of its Ritz vector, and the steps taken."""
    V = np.zeros((start.size, maxdim + 1))
    V[:, 0] = start / np.linalg.norm(start)
    alpha, beta, step, warm = np.zeros(maxdim), np.zeros(maxdim), None, None
    for k in range(maxdim):
        w = op(V[:, k])
        if k > 0:
            w -= beta[k - 1] * V[:, k - 1]
        alpha[k] = w @ V[:, k]
        w -= alpha[k] * V[:, k]
        beta[k] = np.linalg.norm(w)
        V[:, k + 1] = w / beta[k]
        if (k + 1) % 3 and k < maxdim - 1:
            continue
        ev, Y = np.linalg.eigh(np.diag(alpha[:k + 1]) + np.diag(beta[:k], 1) + np.diag(beta[:k], -1))
        if abs(beta[k] * Y[k, -1]) >= 1e-4 and k < maxdim - 1:
            continue
        z1, z2 = V[:, :k + 1] @ Y[:, -1], V[:, :k + 1] @ Y[:, -2]
        warm, m2 = op(z1), op(z2)
        r1, r2 = np.linalg.norm(warm - ev[-1] * z1), np.linalg.norm(m2 - ev[-1] * z2)
        gap = ev[-1] - ev[-2] - r2
        gamma = min(r1, r1 * r1 / (gap if gap > 0 else 1e-16))
        step = np.inf if gamma + ev[-1] <= 0 else 1.0 / (gamma + ev[-1])
        if gamma < 1e-3 or gamma + ev[-1] <= 0.5:
            break
    return step, warm, k + 1


@pytest.mark.parametrize("n", [64, 300, 700, 2001])
def test_consecutive_bounds(gpu_lib, n):
    L, ip = _lib.load(), C.POINTER(C.c_int)
    rng = np.random.default_rng(n)
    G = rng.standard_normal((n, n))
    Cm = np.eye(n) + G @ G.T / n
    H = {kind: _direction(kind, n, rng) for kind in KINDS[:-1]}
    H["spike"] = np.diag(np.r_[100.0, rng.uniform(0.1, 1.0, n - 1)])
    inst = instances._assemble("bounds", n, instances._dense_columns(n, [Cm] + [H[k] for k in KINDS]), np.zeros(len(KINDS)))
    Li = np.linalg.inv(np.linalg.cholesky(Cm))
    raw = _raw_vector(n)
    ints = [np.ascontiguousarray(a, np.int32) for a in (inst.Ap, inst.Ai)]
    user, cone, inside, bound = C.c_void_p(), C.c_void_p(), C.c_int(), C.c_double()
    assert L.HUserDataCreate(C.byref(user)) == 0
    L.HUserDataSetConeData(user, DENSE_SDP, len(KINDS), n, *[a.ctypes.data_as(ip) for a in ints], api._dp(inst.Ax))
    assert L.HConeCreate(C.byref(cone)) == 0 and L.HConeSetData(cone, user) == 0
    try:
        assert L.HConeProcData(cone) == 0 and L.HConePresolveData(cone) == 0
        L.HConeSetStart(cone, 0.0)
        y = np.zeros(len(KINDS))
        assert L.HConeCheckIsInterior(cone, 1.0, api._dp(y), C.byref(inside)) == 0 and inside.value
        starts, taken = [raw], []
        for kind in ORDER:
            dy = np.array([1.0 if k == kind else 0.0 for k in KINDS])
            assert L.HConeRatioTest(cone, 0.0, api._dp(dy), 0.0, VAR, C.byref(bound)) == 0
            op = lambda x: Li @ (H[kind] @ (Li.T @ x))   # -L^-1 dS L^-T with dS = -H
            got = [_bound(op, s) for s in starts]
            step, warm, steps = min(got, key=lambda g: abs(g[0] - bound.value))
            assert bound.value == pytest.approx(step, rel=1e-8), (kind, taken)
            taken.append(steps)
            starts = [warm + 1e-3 * raw, -warm + 1e-3 * raw]
        # the schedule met both a bound that was over at once and one after it that was not
        assert min(taken) <= 6 and any(b > a + 6 for a, b in zip(taken, taken[1:]))
    finally:
        L.HConeDestroy(C.byref(cone))
        L.HUserDataDestroy(C.byref(user))
