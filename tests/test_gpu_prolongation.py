"""GPU: the prolongation and fine-to-coarse correction passes for every
interpol_type and at entry counts below, at and above their 128-thread
blocks, FP64 against the oracle bit for bit."""
import numpy as np
import pytest

import oracle
from ramses_b200 import ics, mesh, runtime

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


def box_tree(size):
    """Level 4 complete, level 5 a box of size[0] x size[1] x size[2] octs;
    (tree, prolongation entries, correction targets) of level 5."""
    lo = np.array([3, 2, 1])

    def refine(level, cells):
        return np.all((cells >= lo) & (cells < lo + np.array(size)), axis=1)
    tree = mesh.build_tree(4, 5, refine, nexpand=0)
    octs = {tuple(x) for x in tree.coords[5].tolist()}
    assert len(octs) == size[0] * size[1] * size[2]
    near = {tuple(((np.array(x) + np.array(d) - 1) % 16).tolist()) for x in octs for d in np.ndindex(3, 3, 3)}
    nc = tree.nbor[:, tree.active[5] - 1]
    return tree, len(near - octs), len(np.unique(nc[tree.son[nc - 1] == 0]))


@pytest.mark.parametrize("size,entries,targets", [((1, 1, 1), 26, 6), ((2, 2, 8), 128, 72), ((4, 4, 6), 192, 128),
                                                  ((2, 4, 13), 256, 172)])
@pytest.mark.parametrize("device", [False, True])
def test_counts_at_the_block_size(cuda_lib, oracle_lib, size, entries, targets, device):
    """Entry counts below, at and above multiples of 128, and correction
    targets whose five values fill whole blocks or not, through the host- and
    the device-scheduled coarse steps."""
    tree, n_entries, n_targets = box_tree(size)
    assert (n_entries, n_targets) == (entries, targets)
    _, hp, _ = sedov_amr(3, 3, slope_type=2)

    def prim(x):
        q = np.zeros((5, len(x)))
        q[0] = 1.0 + 0.3 * np.cos(9 * x[:, 0]) * np.sin(5 * x[:, 1])
        q[1], q[2], q[3] = 0.5 * np.sin(7 * x[:, 2]), 0.4, -0.3 * np.cos(6 * x[:, 0])
        q[4] = 1.0 + 0.5 * np.sin(8 * x[:, 1] + 3 * x[:, 2])
        return q
    u = ics.fill_all_levels(tree, prim, hp.gamma)
    orc = oracle.OracleRun(tree, hp, u)
    with runtime.Solver(tree, hp, uold=u) as s:
        for _ in range(2):
            orc.coarse_step()
            if device:
                assert s.run(max_steps=1) == 1
            else:
                s.coarse_step()
        np.testing.assert_array_equal(s.download_state(), orc.uold)
