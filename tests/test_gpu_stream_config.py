"""GPU: the default z-streaming configuration and every work-item extent give
the same state as the oct tiles (FP64 bit for bit) and, in FP32-mixed, the
same bits for every extent of one column shape."""
import numpy as np
import pytest

from ramses_b200 import runtime

from helpers import turbulent_uniform

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level", [3, 4, 5, 6, 7])
def test_default_equals_tiles(cuda_lib, level):
    tree, hp, u = turbulent_uniform(level)
    with runtime.Solver(tree, hp, uold=u) as a, runtime.Solver(tree, hp, uold=u) as b:
        a.set_uniform_method("tiles")
        a.uniform_run(2)
        b.uniform_run(2)
        info = b.uniform_info()
        n = 2 ** level
        assert info["method"] == "stream" and n % info["hz"] == 0 and info["items"] >= 1
        np.testing.assert_array_equal(a.download_state(), b.download_state())
        assert a.t == b.t


@pytest.mark.parametrize("hz", [2, 8, 16, 64])
def test_mixed_extent_changes_nothing(cuda_lib, hz):
    tree, hp, u = turbulent_uniform(6)
    with runtime.Solver(tree, hp, precision="mixed", uold=u) as a, \
            runtime.Solver(tree, hp, precision="mixed", uold=u) as b:
        a.uniform_run(3)
        b.uniform_run(0)
        b.set_stream_shape(6, hz)
        b.uniform_run(3)
        np.testing.assert_array_equal(a.download_state(), b.download_state())
        assert a.t == b.t
