"""The one-launch Lanczos step bound of small blocks (order <= 96) at the edges of its 8-row
blocks, and of blocks just above, against a NumPy restatement of the reference's estimator
(linalg/hdsdp_lanczos.c:33-53, :161-292) from the same start vector. Bar: 1e-8 relative, that of
the step parity tests; the bound never exceeds the exact step 1 / lambda_max(-L^-1 dS L^-T)."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from hdsdp_b200 import api, instances
from oracle import kernels_ref as K

pytestmark = pytest.mark.gpu


def _start_vector(n):
    libc = C.CDLL(None)
    libc.srand(n)
    v = np.zeros(n)
    for i in range(n):
        libc.srand(libc.rand())
        r1, r2 = libc.rand() % 1627, libc.rand() % 2
        v[i] = np.sqrt(np.sqrt(float(r1))) * (r2 - 0.5)
    return v / np.linalg.norm(v)


def lanczos_step(S, dS, maxdim=30):
    """The estimator's step bound for the operator -L^-1 dS L^-T."""
    n = S.shape[0]
    Li = np.linalg.inv(np.linalg.cholesky(S))
    op = lambda x: Li @ (-(dS @ (Li.T @ x)))
    V = np.zeros((n, maxdim + 1))
    V[:, 0] = _start_vector(n)
    alpha, beta, step = np.zeros(maxdim), np.zeros(maxdim), None
    for k in range(maxdim):
        w = op(V[:, k])
        if k > 0:
            w -= beta[k - 1] * V[:, k - 1]
        alpha[k] = w @ V[:, k]
        w -= alpha[k] * V[:, k]
        beta[k] = np.linalg.norm(w)
        V[:, k + 1] = w / beta[k] if beta[k] > 0 else 0.0
        if (k + 1) % 3 and k < maxdim - 1 and beta[k] > 0:
            continue
        ev, Y = np.linalg.eigh(np.diag(alpha[:k + 1]) + np.diag(beta[:k], 1) + np.diag(beta[:k], -1))
        if abs(beta[k] * Y[k, -1]) >= 1e-4 and k < maxdim - 1:
            continue
        z1, z2 = V[:, :k + 1] @ Y[:, -1], V[:, :k + 1] @ Y[:, -2]
        r1, r2 = np.linalg.norm(op(z1) - ev[-1] * z1), np.linalg.norm(op(z2) - ev[-1] * z2)
        gap = ev[-1] - ev[-2] - r2
        gamma = min(r1, r1 * r1 / (gap if gap > 0 else 1e-16))
        step = np.inf if gamma + ev[-1] <= 0 else 1.0 / (gamma + ev[-1])
        if gamma < 1e-3 or gamma + ev[-1] <= 0.5 or beta[k] == 0:
            break
    return step


@pytest.mark.parametrize("n", [3, 7, 8, 9, 16, 17, 31, 40, 41, 63, 64, 65, 88, 89, 95, 96, 97, 128, 131, 200, 255, 257,
                               300, 440, 456, 457, 600])
def test_step_bound(gpu_lib, n):
    rng = np.random.default_rng(n)
    G = rng.standard_normal((n, n))
    Cm = np.eye(n) + G @ G.T / n
    mats = [Cm]
    for i in range(n):
        E = np.zeros((n, n))
        E[i, i] = 1.0
        mats.append(E)
    inst = instances._assemble("bound", n, instances._dense_columns(n, mats), np.zeros(n))
    y = -rng.uniform(0.0, 0.5, n)
    dy = rng.uniform(0.1, 1.0, n)
    S, dS = K.dual_slack(Cm, mats[1:], y), -np.diag(dy)
    step, logdet = api.ratio_probe(inst, y, 0.0, dy, 0.0)
    assert step <= K.max_step(S, dS) * (1 + 1e-9)
    assert step == pytest.approx(lanczos_step(S, dS), rel=1e-8)
    assert logdet == pytest.approx(np.linalg.slogdet(S)[1], rel=1e-12, abs=1e-11)
