"""What a user has this library do, as cases that can be timed.

The unit of work of an interior-point host is the dual-scaling iteration. ``iterate`` cases
drive the conic callback interface (include/hdsdp_conic.h) as such a host does, two iterations
a pass: interior check (assembly and Cholesky factor of the dual slack), log barrier, Schur
complement and its right-hand sides, factorisation, Schur solves, Lanczos step bound, a line
search point, and a corrector at the accepted point; small problems also recover the primal.
``solve`` cases are whole HDSDPOptimize calls under an iteration budget, and ``schur`` cases
one Schur complement in split precision (BF16x3 products on the tensor cores).

Problems are those of hdsdp_b200/instances.py, with other seeds and sizes.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from hdsdp_b200 import _lib, api, instances

DENSE_SDP, LP, SCALAR_BOUND = 4, 1, 3
VAR, CHECK = 0, 1
INFEASIBLE, CORRECTOR, HOMOGENEOUS = 0, 1, 2
STEPS = 2          # dual-scaling iterations a pass
MU = 1.0
INT_PARAM_MAXITER = 0

_vp, _ip, _dp = C.c_void_p, C.POINTER(C.c_int), C.POINTER(C.c_double)


def listed():
    return [
        # the smallest problems: every operation is a launch and a wait
        {"name": "maxcut n50", "kind": "iterate", "family": "maxcut", "n": 50, "deg": 8, "resi": -1.0, "kkt": INFEASIBLE, "primal": True},
        # MaxCut on a 200-vertex graph, infeasible start (a dual residual in S)
        {"name": "maxcut n200", "kind": "iterate", "family": "maxcut", "n": 200, "deg": 10, "resi": -1.0, "kkt": INFEASIBLE, "primal": True},
        # MaxCut above the order from which trial points are factored sparsely; odd order
        {"name": "maxcut n2001", "kind": "iterate", "family": "maxcut", "n": 2001, "deg": 10, "resi": 0.0, "kkt": INFEASIBLE, "primal": False},
        # the largest single-block workload: 40,000 edges, M as large as S
        {"name": "maxcut n8000", "kind": "iterate", "family": "maxcut", "n": 8000, "deg": 10, "resi": 0.0, "kkt": INFEASIBLE, "primal": False},
        # Lovasz theta, small, in the self-dual embedding (the extra products with C)
        {"name": "theta n100 embedding", "kind": "iterate", "family": "theta", "n": 100, "p": 0.1, "resi": -1.0, "kkt": HOMOGENEOUS, "primal": True},
        # Lovasz theta at its workload size: M (about 4,500 rows) far larger than S
        {"name": "theta n300", "kind": "iterate", "family": "theta", "n": 300, "p": 0.1, "resi": 0.0, "kkt": INFEASIBLE, "primal": True},
        # rank-one constraints at odd sizes, infeasible start
        {"name": "rank1 n333 m517", "kind": "iterate", "family": "rank1", "n": 333, "m": 517, "density": 0.1, "resi": -1.0, "kkt": INFEASIBLE, "primal": True},
        # the benchmark workload: 2,000 rank-one constraints of support 100 in order 1,000
        {"name": "rank1 n1000 m2000", "kind": "iterate", "family": "rank1", "n": 1000, "m": 2000, "density": 0.1, "resi": 0.0, "kkt": INFEASIBLE, "primal": False},
        # general dense coefficient matrices
        {"name": "dense n80 m40", "kind": "iterate", "family": "dense", "n": 80, "m": 40, "resi": 0.0, "kkt": INFEASIBLE, "primal": True},
        # dense and sparse cones and an LP cone over shared constraints
        {"name": "blocks m800 lp", "kind": "iterate", "family": "blocks", "dims": "200,150,100,50", "local": "300,200,150,100", "couple": 50, "lp": 60, "resi": 0.0,
         "kkt": INFEASIBLE, "primal": False},
        # a whole solve from data on the host, stopped by its iteration budget
        {"name": "solve maxcut n200", "kind": "solve", "family": "maxcut", "n": 200, "deg": 10, "maxiter": 6},
        # one Schur complement in split precision, from data on the host
        {"name": "schur split n600 m900", "kind": "schur", "family": "rank1", "n": 600, "m": 900, "density": 0.1},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["maxcut", "maxcut", "theta", "rank1", "rank1", "dense", "blocks", "solve"])
    resi = rng.choice([0.0, -1.0])
    c = {"kind": "iterate", "family": family, "resi": resi, "kkt": INFEASIBLE, "primal": False}
    if family == "maxcut":
        c.update(n=_log_int(rng, 40, 4500), deg=rng.randint(6, 14))
        c["primal"] = c["n"] <= 400
    elif family == "theta":
        c.update(n=_log_int(rng, 30, 300), p=round(rng.uniform(0.05, 0.1), 4), kkt=rng.choice([INFEASIBLE, HOMOGENEOUS]), primal=True)
    elif family == "rank1":
        n = _log_int(rng, 40, 1000)
        c.update(n=n, m=min(2000, max(20, int(n * rng.uniform(0.8, 2.0)))), density=0.1, primal=n <= 400)
        if rng.random() < 0.25:
            c = {"kind": "schur", "family": "rank1", "n": min(n, 700), "m": min(c["m"], 1000), "density": 0.1}
    elif family == "dense":
        c.update(n=_log_int(rng, 20, 120), m=rng.randint(10, 60), primal=True)
    elif family == "blocks":
        k = rng.randint(2, 4)
        dims = sorted((_log_int(rng, 15, 220) for _ in range(k)), reverse=True)
        c.update(dims=",".join(map(str, dims)), local=",".join(str(int(n * rng.uniform(0.8, 1.5))) for n in dims), couple=rng.randint(4, 40), lp=rng.choice([0, rng.randint(8, 80)]))
    else:
        return {"kind": "solve", "family": "maxcut", "n": _log_int(rng, 100, 700), "deg": rng.randint(8, 14), "maxiter": rng.randint(4, 6)}
    return c


# ---- problems -----------------------------------------------------------------------------


def _rank_one_vectors(n, m, density, rng):
    """Supports (m x k, increasing) and values of the vectors a_i of A_i = a_i a_i^T."""
    k = max(1, int(round(density * n)))
    supp = np.sort(np.argsort(rng.random((m, n)), axis=1)[:, :k], axis=1)
    return supp, rng.standard_normal((m, k))


def _rank_one(n, m, density, seed):
    rng = np.random.default_rng(seed)
    supp, a = _rank_one_vectors(n, m, density, rng)
    k = supp.shape[1]
    J, I = np.triu_indices(k)  # column by column: packed indices increase
    idx = instances.pack_idx(n, supp[:, I], supp[:, J])
    val = a[:, I] * a[:, J]
    G = rng.standard_normal((n, 20))
    Ga = np.einsum("mk,mkr->mr", a, G[supp])
    b = (a * a).sum(1) + (Ga * Ga).sum(1) / n
    r, c = np.tril_indices(n, -1)
    keep = rng.random(r.size) < 0.01
    diag = np.arange(n)
    ci = np.concatenate([instances.pack_idx(n, diag, diag), instances.pack_idx(n, r[keep], c[keep])])
    cv = np.concatenate([np.ones(n), rng.uniform(-0.1, 0.1, size=int(keep.sum()))])
    o = np.argsort(ci)
    Ap = np.concatenate([[0], ci.size + idx.shape[1] * np.arange(m + 1)])
    inst = instances.SDPInstance("rank_one", n, m, Ap.astype(np.int32), np.concatenate([ci[o], idx.ravel()]).astype(np.int32),
                                 np.concatenate([cv[o], val.ravel()]), b)
    return inst, supp, a


def _maxcut(case, seed):
    n = case["n"]
    edges = min(n * case["deg"] // 2, n * (n - 1) // 4)
    return instances.maxcut(n, seed=seed, n_edges=edges, weights=(0.5, 1.5))


def _problem(case, seed):
    """(cones as (type, dim, Ap, Ai, Ax), b, a strictly feasible dual point)."""
    rng = np.random.default_rng(seed + 1)
    family = case["family"]
    if family == "blocks":
        prob = instances.multiblock([int(x) for x in case["dims"].split(",")], [int(x) for x in case["local"].split(",")], case["couple"], n_lp=case["lp"], seed=seed)
        cones = [(DENSE_SDP if kind == "sdp" else LP, dim, Ap, Ai, Ax) for kind, dim, Ap, Ai, Ax in prob.cones]
        return cones, prob.b, 0.01 * rng.uniform(-1.0, 1.0, prob.m)
    if family == "maxcut":
        inst = _maxcut(case, seed)
        rows, vals = inst.column(0)
        diag = np.zeros(inst.n)
        start = instances.pack_idx(inst.n, np.arange(inst.n), np.arange(inst.n))
        at = np.searchsorted(start, rows)
        hit = start[np.minimum(at, inst.n - 1)] == rows
        diag[at[hit]] = vals[hit]
        y = 2.0 * diag - rng.uniform(0.5, 1.5, inst.n)  # S = C - diag(y) is diagonally dominant
    elif family == "theta":
        r, c = np.tril_indices(case["n"], -1)
        pick = np.sort(rng.choice(r.size, size=int(case["p"] * r.size), replace=False))
        inst = instances.lovasz_theta_graph(case["n"], list(zip(r[pick].tolist(), c[pick].tolist())))
        y = rng.uniform(-0.5, 0.5, inst.m)
        y[0] = -(1.5 * inst.n + 10.0)
    elif family == "rank1":
        inst = _rank_one(case["n"], case["m"], case["density"], seed)[0]
        y = -rng.uniform(0.001, 0.02, inst.m)
    else:
        inst = instances.dense_coeff(case["n"], case["m"], seed=seed)
        y = (0.02 / case["n"]) * rng.uniform(-1.0, 1.0, inst.m)
    return [(DENSE_SDP, inst.n, inst.Ap, inst.Ai, inst.Ax)], inst.b, y


# ---- a host that drives the cones and the Schur complement --------------------------------


def _p(a):
    return a.ctypes.data_as(_dp)


class _Host:
    def __init__(self, cones, b, y, case):
        L = self.L = _lib.load()
        self.b, self.y0, self.case = np.ascontiguousarray(b), np.ascontiguousarray(y), case
        self.m = m = b.size
        self.keep, self.users, self.cones = [], [], []
        lo_up = np.array([-1e7, 1e7])
        none = np.zeros(1, np.int32)
        for kind, dim, Ap, Ai, Ax in cones + [(SCALAR_BOUND, m, none, none, lo_up)]:
            arrays = [np.ascontiguousarray(Ap, np.int32), np.ascontiguousarray(Ai, np.int32), np.ascontiguousarray(Ax, np.float64)]
            user, cone = _vp(), _vp()
            self._ok(L.HUserDataCreate(C.byref(user)))
            L.HUserDataSetConeData(user, kind, m, dim, arrays[0].ctypes.data_as(_ip), arrays[1].ctypes.data_as(_ip), _p(arrays[2]))
            self._ok(L.HConeCreate(C.byref(cone)))
            self._ok(L.HConeSetData(cone, user))
            self._ok(L.HConeProcData(cone))
            self._ok(L.HConePresolveData(cone))
            L.HConeSetStart(cone, case["resi"])
            self.keep.append(arrays)
            self.users.append(user)
            self.cones.append(cone)
        self.bound = self.cones[-1]
        self.main = self.cones[:-1]
        self.n = cones[0][1]
        self.handles = (_vp * len(self.main))(*[c.value for c in self.main])
        self.kkt = _vp()
        self._ok(L.HKKTCreate(C.byref(self.kkt)))
        self._ok(L.HKKTInit(self.kkt, m, len(self.main), self.handles))

    @staticmethod
    def _ok(code):
        if code != 0:
            raise RuntimeError("a library call returned %d" % code)

    def check(self, y, buffer=VAR):
        """S(y) positive definite in every cone, and the log barrier there."""
        inside, value, total = C.c_int(), C.c_double(), 0.0
        for c in self.cones:
            if buffer == VAR:
                self._ok(self.L.HConeCheckIsInterior(c, 1.0, _p(y), C.byref(inside)))
            else:
                self._ok(self.L.HConeCheckIsInteriorExpert(c, 1.0, -1.0, _p(y), -self.case["resi"], buffer, C.byref(inside)))
            if not inside.value:
                raise RuntimeError("the point is not interior")
            self._ok(self.L.HConeGetLogBarrier(c, 0.0, None, buffer, C.byref(value)))
            if c is not self.bound:
                total += value.value
        return total

    def build(self, kind):
        self._ok(self.L.HKKTBuildUp(self.kkt, kind))
        self._ok(self.L.HKKTBuildUpExtraCone(self.kkt, self.bound, kind))
        vectors = [np.zeros(self.m) for _ in range(3)]
        scalars = [C.c_double() for _ in range(4)]
        self.L.HKKTExport(self.kkt, *[_p(v) for v in vectors], *[C.byref(s) for s in scalars])
        return vectors, np.array([s.value for s in scalars])

    def solve(self, rhs):
        out = np.zeros(self.m)
        self._ok(self.L.HKKTSolve(self.kkt, _p(rhs), _p(out)))
        return out

    def step(self, dy):
        bound, step = C.c_double(), math.inf
        for c in self.main:
            self._ok(self.L.HConeRatioTest(c, 0.0, _p(dy), 0.0, VAR, C.byref(bound)))
            step = min(step, bound.value)
        return step

    def iterate(self):
        out = {"steps": []}
        y, logdet = self.y0, []
        for it in range(STEPS):
            r = {}
            logdet.append(self.check(y))
            (asinv, asinvrd, asinvcs), scalars = self.build(self.case["kkt"])
            self._ok(self.L.HKKTFactorize(self.kkt))
            d1, d2 = self.solve(self.b), self.solve(asinv)
            dy = d1 / MU - d2
            r.update(asinv=asinv, dy=dy)
            if self.case["resi"]:
                r.update(asinvrd=asinvrd, d3=self.solve(asinvrd))
            if self.case["kkt"] == HOMOGENEOUS:
                r.update(asinvcs=asinvcs, d4=self.solve(asinvcs), scalars=scalars)
            alpha = 1.0 / (1.0 + math.sqrt(float((self.b / MU - asinv) @ dy)))  # inside the Dikin ellipsoid
            out["steps"].append(self.step(dy))
            logdet.append(self.check(y + alpha * dy, CHECK))
            y = y + 0.8 * alpha * dy
            logdet.append(self.check(y))
            (asinv, _, _), _ = self.build(CORRECTOR)
            dc = self.solve(self.b / MU - asinv)
            out["steps"].append(self.step(dc))
            y = y + (0.5 / (1.0 + math.sqrt(abs(float((self.b / MU - asinv) @ dc))))) * dc
            r.update(corrector=dc, y=y)
            out["it%d" % it] = r
        out["logdet"] = np.array(logdet)
        if self.case["primal"]:
            X = np.zeros((self.n, self.n))
            self.L.HConeGetPrimal(self.main[0], MU, _p(self.y0), _p(out["it0"]["dy"]), _p(X), None)
            out["X"] = X
        return out

    def __del__(self):
        if getattr(self, "kkt", None):
            self.L.HKKTDestroy(C.byref(self.kkt))
        for c in getattr(self, "cones", []):
            self.L.HConeDestroy(C.byref(c))
        for u in getattr(self, "users", []):
            self.L.HUserDataDestroy(C.byref(u))


def prepare(case, seed):
    if case["kind"] == "solve":
        return {"case": case, "inst": _maxcut(case, seed)}
    if case["kind"] == "schur":
        inst = _rank_one(case["n"], case["m"], case["density"], seed)[0]
        return {"case": case, "inst": inst, "y": -np.random.default_rng(seed + 1).uniform(0.001, 0.02, inst.m)}
    return {"case": case, "host": _Host(*_problem(case, seed), case)}


def run(state):
    case = state["case"]
    if case["kind"] == "solve":
        r = api.solve(state["inst"], params={INT_PARAM_MAXITER: case["maxiter"]})
        return {"y": r["y"], "S": r["S"], "dobj": np.array([r["dobj"]]), "iterations": r["iters"]}
    if case["kind"] == "schur":
        return api.schur_probe(state["inst"], state["y"], 0.0, precision=1)
    return state["host"].iterate()


# ---- operations and bytes that a pass cannot do without ------------------------------------


def work(case):
    n = case.get("n", 0)
    m = case.get("m", n)
    factor = lambda k: k ** 3 / 3.0
    if case["kind"] == "solve":
        # per iteration: at least two points factored, one S^-1, M = S^-1 o S^-1, one factor of M
        per = 2 * factor(n) + 2 * factor(n) + n * n + factor(n) + 6.0 * n * n
        return {"bytes": 8.0 * (n * n + 4 * n) + 12.0 * n * case["deg"], "flops": case["maxiter"] * per}
    if case["kind"] == "schur":
        k = max(1, int(round(case["density"] * n)))
        return {"bytes": 12.0 * m * k * (k + 1) / 2 + 8.0 * m * m, "flops": 2 * factor(n) + 2.0 * n * k * m + n * m * (m + 1.0)}
    if case["family"] == "blocks":
        dims, local = ([int(x) for x in case[k].split(",")] for k in ("dims", "local"))
        rows = [l + case["couple"] for l in local]
        m = sum(local) + case["couple"]
    else:
        dims, rows = [n], [m]
    if case["family"] == "theta":
        m = rows[0] = int(case["p"] * n * (n - 1) / 2) + 1
    if case["family"] == "maxcut":
        pairs, data = 2.0 * n * n, n * (case["deg"] + 2.0)
    elif case["family"] == "theta":
        pairs, data = 5.0 * m * m / 2, n * (n + 1) / 2 + m
    elif case["family"] == "rank1":
        k = max(1, int(round(case["density"] * n)))
        pairs, data = 2.0 * n * k * m + n * m * (m + 1.0), m * k * (k + 1) / 2
    elif case["family"] == "dense":
        pairs, data = m * (4.0 * n ** 3 + n * n * (m + 1.0)), m * n * (n + 1) / 2
    else:
        pairs, data = sum(10.0 * r * r for r in rows), sum(8.0 * r for r in rows)
    # an iteration: three slacks factored, two inverses, M and its factor, three solves, two step
    # bounds (at least eight products with L^-1, dS and L^-T each)
    per = sum(3 * factor(d) + 4 * factor(d) + 2 * 8 * 4.0 * d * d for d in dims) + pairs + factor(m) + 3 * 2.0 * m * m
    primal = 6.0 * dims[0] ** 3 if case["primal"] else 0.0
    written = 8.0 * (STEPS * 8 * m + (n * n if case["primal"] else 0))
    return {"bytes": 12.0 * data + written, "flops": STEPS * per + primal}


# ---- the same in 64 bits with torch ---------------------------------------------------------


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Exact:
    """C, the A_i and the barrier of one SDP block (as vectors a_i of A_i = a_i a_i^T, or as
    full matrices) or of an LP cone."""

    def __init__(self, cone, m, vectors=None):
        kind, self.n, Ap, Ai, Ax = cone
        self.lp, n, d = kind == LP, cone[1], _device()
        self.U = vectors
        col = np.repeat(np.arange(m + 1), np.diff(Ap))
        if self.lp:
            A = np.zeros((m + 1, n))
            A[col, Ai] = Ax
            A = torch.from_numpy(A).to(d)
            self.C, self.A = A[0], A[1:]
            return
        start = instances.pack_idx(n, np.arange(n), np.arange(n))
        sel = slice(None) if vectors is None else slice(0, Ap[1])
        col, rows, vals = col[sel], np.asarray(Ai)[sel], np.asarray(Ax)[sel]
        j = np.searchsorted(start, rows, side="right") - 1
        i = rows - start[j] + j
        A = torch.zeros((m + 1 if vectors is None else 1, n, n), dtype=torch.float64, device=d)
        col, i, j, v = (torch.from_numpy(np.ascontiguousarray(x)).to(d) for x in (col, i, j, vals))
        A[col, i, j] = v
        A[col, j, i] = v
        self.C, self.A = A[0], A[1:]

    def at(self, y, resi):
        if self.lp:
            self.s = self.C - self.A.T @ y - resi
            return float(self.s.log().sum())
        AY = (self.U * y) @ self.U.T if self.U is not None else torch.einsum("m,mij->ij", y, self.A)
        self.S = self.C - AY - resi * torch.eye(self.n, dtype=torch.float64, device=y.device)
        L = torch.linalg.cholesky(self.S)
        self.W = torch.cholesky_inverse(L)
        return 2.0 * float(L.diagonal().log().sum())

    def vectors(self, resi):
        """<A_i, W>, resi <A_i, W^2>, <A_i, W C W>; <C, W C W>, <C, W>, resi tr(W C W), tr W."""
        if self.lp:
            w = 1.0 / self.s
            return self.A @ w, resi * (self.A @ (w * w)), self.A @ (w * w * self.C), [0.0] * 4
        W, WCW = self.W, self.W @ self.C @ self.W
        if self.U is not None:
            q = lambda Z: (self.U * (Z @ self.U)).sum(0)
        else:
            q = lambda Z: (self.A.reshape(len(self.A), -1) @ Z.reshape(-1))
        return q(W), resi * q(W @ W), q(WCW), [float((self.C * WCW).sum()), float((self.C * W).sum()), resi * float(WCW.trace()), float(W.trace())]

    def schur(self):
        if self.lp:
            Q = self.A / self.s
            return Q @ Q.T
        if self.U is not None:
            G = self.U.T @ self.W @ self.U
            return G * G
        flat = self.A.reshape(len(self.A), -1)
        M = torch.empty((len(self.A), len(self.A)), dtype=torch.float64, device=flat.device)
        for k in range(0, len(self.A), 512):
            M[k:k + 512] = (self.W @ self.A[k:k + 512] @ self.W).reshape(-1, flat.shape[1]) @ flat.T
        return M

    def operator(self, dy):
        return (self.U * dy) @ self.U.T if self.U is not None else torch.einsum("m,mij->ij", dy, self.A)


def exact(case, seed):
    if case["kind"] == "solve":
        return None
    d = _device()
    vectors = None
    if case["family"] == "rank1":
        inst, supp, a = _rank_one(case["n"], case["m"], case["density"], seed)
        U = np.zeros((case["n"], case["m"]))
        U[supp.T, np.arange(case["m"])[None, :]] = a.T
        vectors = torch.from_numpy(U).to(d)
    elif case["family"] == "maxcut":
        vectors = torch.eye(case["n"], dtype=torch.float64, device=d)
    host = lambda t: t.cpu().numpy()
    if case["kind"] == "schur":
        e = _Exact((DENSE_SDP, inst.n, inst.Ap, inst.Ai, inst.Ax), inst.m, vectors)
        y = -np.random.default_rng(seed + 1).uniform(0.001, 0.02, inst.m)
        e.at(torch.from_numpy(y).to(d), 0.0)
        asinv, _, _, _ = e.vectors(0.0)
        return {"M": host(torch.tril(e.schur())), "asinv": host(asinv), "asinvrd": None, "tracesinv": None}
    cones, b, y0 = _problem(case, seed)
    m, resi, homogeneous = b.size, case["resi"], case["kkt"] == HOMOGENEOUS
    blocks = [_Exact(c, m, vectors) for c in cones]
    b, y = torch.from_numpy(b).to(d), torch.from_numpy(np.ascontiguousarray(y0)).to(d)


    def sums():
        a, ard, acs = (sum(x) for x in list(zip(*[e.vectors(resi) for e in blocks]))[:3])
        lo, up = 1.0 / (y + 1e7), 1.0 / (1e7 - y)  # the box -1e7 <= y <= 1e7
        return a + up - lo, ard, acs + 1e7 * (up * up - lo * lo), lo * lo + up * up

    out, logdet = {"steps": [None] * (2 * STEPS)}, []
    for it in range(STEPS):
        logdet.append(sum(e.at(y, resi) for e in blocks))
        asinv, asinvrd, asinvcs, box = sums()
        L = torch.linalg.cholesky(sum(e.schur() for e in blocks) + torch.diag(box))
        solve = lambda v: torch.cholesky_solve(v[:, None], L)[:, 0]
        dy = solve(b) / MU - solve(asinv)
        r = {"asinv": asinv, "dy": dy}
        if it == 0 and case["primal"]:
            e = blocks[0]
            X = MU * (e.W + e.W @ e.operator(dy) @ e.W)
        if resi:
            r.update(asinvrd=asinvrd, d3=solve(asinvrd))
        if homogeneous:
            r.update(asinvcs=asinvcs, d4=solve(asinvcs))
        alpha = 1.0 / (1.0 + math.sqrt(float((b / MU - asinv) @ dy)))
        logdet.append(sum(e.at(y + alpha * dy, resi) for e in blocks))
        y = y + 0.8 * alpha * dy
        logdet.append(sum(e.at(y, resi) for e in blocks))
        asinv = sums()[0]
        dc = solve(b / MU - asinv)
        y = y + (0.5 / (1.0 + math.sqrt(abs(float((b / MU - asinv) @ dc))))) * dc
        r.update(corrector=dc, y=y)
        out["it%d" % it] = {k: host(v) for k, v in r.items()}
        if homogeneous:
            out["it%d" % it]["scalars"] = None
    out["logdet"] = np.array(logdet)
    if case["primal"]:
        out["X"] = None if resi else host(X)
    return out
