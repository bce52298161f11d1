"""GPU: the prolongation and fine-to-coarse correction passes at small and
ragged entry counts (below, at and above their 128-thread blocks), FP64
against the oracle bit for bit."""
import numpy as np
import pytest

import oracle
from ramses_b200 import runtime

from helpers import sedov_amr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("interpol_type", [0, 1, 2, 3])
@pytest.mark.parametrize("levels", [(2, 4), (3, 4), (4, 5)])
def test_prolongation_per_variable(cuda_lib, oracle_lib, levels, interpol_type):
    tree, hp, u = sedov_amr(*levels, interpol_var=0, interpol_type=interpol_type, slope_type=2)
    orc = oracle.OracleRun(tree, hp, u)
    with runtime.Solver(tree, hp, uold=u) as s:
        for _ in range(2):
            orc.coarse_step()
            s.coarse_step()
        np.testing.assert_array_equal(s.download_state(), orc.uold)
