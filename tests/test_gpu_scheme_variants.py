"""GPU: the compiled llf and hll variants (minmod, moncen) of the z-streaming
kernels and the serving batch: FP64 equals the oracle bit for bit, FP32-mixed
stays within its rounding of FP64 and conserves, on the smallest grid that a
column shape fits and on one with several work items per column."""
import numpy as np
import pytest

import oracle
from ramses_b200 import runtime, serve

from helpers import leaf_values, turbulent_uniform

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level", [3, 4, 6])
@pytest.mark.parametrize("slope_type", [1, 2])
@pytest.mark.parametrize("riemann", ["llf", "hll"])
def test_uniform(cuda_lib, oracle_lib, riemann, slope_type, level):
    tree, hp, u = turbulent_uniform(level, riemann=riemann, slope_type=slope_type)
    orc = oracle.OracleRun(tree, hp, u)
    for _ in range(3):
        orc.coarse_step()
    with runtime.Solver(tree, hp, uold=u) as s:
        s.uniform_run(3)
        np.testing.assert_array_equal(s.download_state(), orc.uold)
        assert s.t == orc.t
    with runtime.Solver(tree, hp, precision="mixed", uold=u) as s:
        s.uniform_run(3)
        out = s.download_state()
    cells, ref = leaf_values(tree, orc.uold)
    got, start = out[:, cells - 1], u[:, cells - 1]
    # some hundred FP32 roundings (6e-8 each) per cell and step
    assert np.all(np.linalg.norm(got - ref, axis=1) <= 1e-5 * np.linalg.norm(ref, axis=1))
    assert np.all(np.abs(got.sum(axis=1) - start.sum(axis=1)) <= 1e-13 * np.abs(start).sum(axis=1))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("riemann", ["llf", "hll"])
def test_served_equals_uniform_run(cuda_lib, riemann, precision):
    tree, hp, u = turbulent_uniform(5, riemann=riemann, slope_type=1)
    with runtime.Solver(tree, hp, precision=precision, uold=u) as s:
        s.uniform_run(5)
        ref = serve.dense_from_octree(tree, 5, s.download_state())
    with serve.Server(hp, precision=precision) as srv:
        rid = srv.submit_dense(serve.dense_from_octree(tree, 5, u), max_steps=5)
        srv.drain()
        np.testing.assert_array_equal(srv.results[rid], ref)
