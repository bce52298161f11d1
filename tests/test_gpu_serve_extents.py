"""GPU: the z extents of a serving round follow its members; a problem's
result must not: alone, in a small batch and in a batch that joins and shrinks
while it runs, for grids whose extents are cut by the cap or by nz."""
import numpy as np
import pytest

from ramses_b200 import serve
from ramses_b200.params import HydroParams

pytestmark = pytest.mark.gpu


def state(n, seed):
    rng = np.random.default_rng(seed)
    u = np.zeros((5, n, n, n))
    u[0] = 1.0 + 0.3 * rng.random((n, n, n))
    u[1:4] = 0.2 * u[0] * (rng.random((3, n, n, n)) - 0.5)
    u[4] = 2.0 + rng.random((n, n, n)) + 0.5 * (u[1:4] ** 2).sum(0) / u[0]
    return u


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("riemann", ["hllc", "llf"])
@pytest.mark.parametrize("sizes", [(16, 48), (32, 32, 64), (16, 80, 48, 64)])
def test_result_independent_of_the_round(cuda_lib, sizes, riemann, precision):
    hp = HydroParams(gamma=1.4, riemann=riemann, slope_type=1, courant_factor=0.8)
    probs = [state(n, i) for i, n in enumerate(sizes)]
    alone = []
    for i, u in enumerate(probs):
        with serve.Server(hp, precision=precision) as srv:
            rid = srv.submit_dense(u, max_steps=5 + 3 * i, outflow_mask=i % 2)
            srv.drain()
            alone.append(srv.results[rid])
    with serve.Server(hp, precision=precision, steps_per_round=3) as srv:
        ids = []
        for i, u in enumerate(probs):
            ids.append(srv.submit_dense(u, max_steps=5 + 3 * i, outflow_mask=i % 2))
            if i % 2:
                srv.progress()
        srv.drain()
        for rid, ref in zip(ids, alone):
            np.testing.assert_array_equal(srv.results[rid], ref)
