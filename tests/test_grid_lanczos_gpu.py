"""The Lanczos step bound above the cluster kernel's order: step matrices that go by their entries
(diagonal, and columns just within the list's length), one with a single column too long, and a
dense one; orders whose columns all stay in shared memory, some of them, and the streamed path.
Oracle and bar as for the smaller orders; at these orders 30 steps may end short of the extreme
eigenvalue, and the estimator then says a little more than the exact step."""
import numpy as np
import pytest

from hdsdp_b200 import api, instances
from test_small_lanczos_gpu import lanczos_step

pytestmark = pytest.mark.gpu


def _direction(kind, n, rng):
    """The constraint matrix that makes the step matrix."""
    H = np.zeros((n, n))
    if kind == "band64":
        for o in range(1, 32):
            H += np.diag(rng.standard_normal(n - o) / 64, -o)
        H[32:, 0] = 0.0
        H[n - 1, 0] = 0.01
    elif kind == "hub":
        H[1:, 0] = rng.standard_normal(n - 1) / n
    elif kind == "dense":
        H = np.tril(rng.standard_normal((n, n)), -1) / n
    return H + H.T + np.diag(rng.uniform(0.1, 1.0, n))


@pytest.mark.parametrize("kind", ["diag", "band64", "hub", "dense"])
@pytest.mark.parametrize("n", [457, 700, 1185, 1500, 2001, 2048, 2049])
def test_step_bound(gpu_lib, n, kind):
    rng = np.random.default_rng(n)
    G = rng.standard_normal((n, n))
    Cm = np.eye(n) + G @ G.T / n
    H = _direction(kind, n, rng)
    inst = instances._assemble("bound", n, instances._dense_columns(n, [Cm, H]), np.zeros(1))
    y, dy = np.array([-0.25]), np.array([1.0])
    S, dS = Cm + 0.25 * H, -H
    step, logdet = api.ratio_probe(inst, y, 0.0, dy, 0.0)
    assert step == pytest.approx(lanczos_step(S, dS), rel=1e-8)
    assert logdet == pytest.approx(np.linalg.slogdet(S)[1], rel=1e-12, abs=1e-11)


@pytest.mark.parametrize("n,kind", [(3000, "hub"), (3000, "dense"), (4097, "diag"), (4097, "hub")])
def test_step_bound_product_by_product(gpu_lib, n, kind):
    """Where each product is a launch: four warps a column below order 4096, one above."""
    test_step_bound(gpu_lib, n, kind)
