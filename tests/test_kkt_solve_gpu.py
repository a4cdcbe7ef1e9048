"""The Schur solve in one launch, on the cluster (up to order 456) and on the grid, at the edges of
their splits, against the Schur matrix itself."""
import ctypes as C

import numpy as np
import pytest

from hdsdp_b200 import _lib, instances

pytestmark = pytest.mark.gpu

_vp = C.c_void_p


def _p(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


@pytest.mark.parametrize("m", [5, 16, 17, 200, 449, 456, 457, 593, 700, 2001, 2049, 3100])
def test_schur_solve(m):
    L = _lib.load()
    inst = instances.maxcut(m, seed=m, n_edges=2 * m if m > 16 else m, weights=(0.5, 1.5))
    rng = np.random.default_rng(m)
    ints = [np.ascontiguousarray(a, np.int32) for a in (inst.Ap, inst.Ai)]
    user, cone, kkt, inside = _vp(), _vp(), _vp(), C.c_int()
    try:
        assert L.HUserDataCreate(C.byref(user)) == 0
        L.HUserDataSetConeData(user, 4, m, m, *[a.ctypes.data_as(C.POINTER(C.c_int)) for a in ints], _p(inst.Ax))
        assert L.HConeCreate(C.byref(cone)) == 0
        assert L.HConeSetData(cone, user) == 0
        assert L.HConeProcData(cone) == 0
        assert L.HConePresolveData(cone) == 0
        L.HConeSetStart(cone, 0.0)
        assert L.HKKTCreate(C.byref(kkt)) == 0
        cones = (_vp * 1)(cone.value)   # kept by the KKT object
        assert L.HKKTInit(kkt, m, 1, cones) == 0
        y = -rng.uniform(30.0, 40.0, m)
        assert L.HConeCheckIsInterior(cone, 1.0, _p(y), C.byref(inside)) == 0 and inside.value
        assert L.HKKTBuildUp(kkt, 0) == 0
        M = np.zeros((m, m))            # its lower triangle, column-major
        assert L.HKKTGetMatrix(kkt, _p(M)) == 0
        M = M + np.triu(M, 1).T
        assert L.HKKTFactorize(kkt) == 0
        for k in range(2):   # the second one reuses the exchange buffers
            b, x = rng.standard_normal(m), np.empty(m)
            assert L.HKKTSolve(kkt, _p(b), _p(x)) == 0
            # refined once: residual of a backward stable solve, |M|_2 <= |M|_1
            assert np.linalg.norm(b - M @ x) <= 4 * np.sqrt(m) * 2.0 ** -52 * np.abs(M).sum(0).max() * np.linalg.norm(x)
    finally:
        for f, h in ((L.HKKTDestroy, kkt), (L.HConeDestroy, cone), (L.HUserDataDestroy, user)):
            if h.value:
                f(C.byref(h))
