"""GPU: the device-scheduled coarse steps (rb_run) with subcycling patterns
that do and do not let the finest level alternate its two buffers, against the
host-scheduled coarse steps and the oracle, FP64 bit for bit."""
import dataclasses

import numpy as np
import pytest

import oracle
from ramses_b200 import ics, mesh, runtime
from ramses_b200.params import HydroParams

from helpers import oct_cells, sedov_amr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("levels", [(3, 3), (3, 4), (3, 6)])
@pytest.mark.parametrize("pattern", [(2, 2), (1, 1), (1, 2), (2, 1)])
def test_subcycling_patterns(cuda_lib, oracle_lib, levels, pattern):
    """pattern: nsubcycle of the even and the odd levels; runs in chunks of
    one, three and a stop in the middle of a graph of eight."""
    tree, hp, u = sedov_amr(*levels)
    ns = [pattern[i % 2] for i in range(33)]
    orc = oracle.OracleRun(tree, hp, u, nsubcycle=ns)
    with runtime.Solver(tree, hp, nsubcycle=ns, uold=u) as s:
        for n in (1, 3):
            assert s.run(max_steps=n) == n
            for _ in range(n):
                orc.coarse_step()
            np.testing.assert_array_equal(s.download_state(), orc.uold)
            assert s.t == orc.t
        t_end = s.t * 1.5
        steps = s.run(t_end=t_end, max_steps=50)
        while orc.t < t_end:
            orc.coarse_step()
            steps -= 1
        assert steps == 0
        np.testing.assert_array_equal(s.download_state(), orc.uold)
        assert s.t == orc.t
        # the finest level's unew holds the state, as after set_uold
        lf = max(l for l in range(1, tree.nlevelmax + 1) if tree.noct(l))
        g = tree.active[lf].astype(np.int64)
        cells = (tree.ncoarse + np.arange(8)[:, None] * tree.ngridmax + g[None, :] - 1).ravel()
        np.testing.assert_array_equal(s.download_unew()[:, cells], orc.uold[:, cells])


@pytest.mark.parametrize("pressure_fix", [False, True])
@pytest.mark.parametrize("stop", ["max_steps", "t_end"])
def test_run_of_no_steps_changes_nothing(cuda_lib, oracle_lib, stop, pressure_fix):
    """A run that is over before it starts leaves uold and unew as they are,
    the levels below levelmin included, which need not be the restriction of
    the finer ones; the next run's step restricts them."""
    tree, hp, u = sedov_amr(3, 5)
    hp.pressure_fix, hp.beta_fix = pressure_fix, 0.5 if pressure_fix else 0.0
    u = u.copy()
    low = np.concatenate([(tree.ncoarse + np.arange(8)[:, None] * tree.ngridmax
                           + tree.active[l].astype(np.int64)[None, :] - 1).ravel() for l in (1, 2)])
    u[:, low] *= 1.25
    unew = u * 1.5
    orc = oracle.OracleRun(tree, hp, u)
    with runtime.Solver(tree, hp, uold=u) as s:
        s.upload_unew(unew)
        assert (s.run(max_steps=0) if stop == "max_steps" else s.run(t_end=s.t, max_steps=5)) == 0
        np.testing.assert_array_equal(s.download_state(), u)
        np.testing.assert_array_equal(s.download_unew(), unew)
        assert s.run(max_steps=1) == 1
        orc.coarse_step()
        cells = oct_cells(tree) - 1
        np.testing.assert_array_equal(s.download_state()[:, cells], orc.uold[:, cells])


@pytest.mark.parametrize("levels", [(3, 4), (3, 6)])
@pytest.mark.parametrize("pattern", [(2, 2), (1, 1), (1, 2), (2, 1)])
def test_subcycling_patterns_pressure_fix(cuda_lib, oracle_lib, levels, pattern):
    """set_unew with divu and enew runs where amr_step has it, at the start
    of each step of a level with finer octs, whatever the pattern."""
    tree, hp, u = sedov_amr(*levels)
    hp.pressure_fix, hp.beta_fix = True, 0.5
    ns = [pattern[i % 2] for i in range(33)]
    orc = oracle.OracleRun(tree, hp, u, nsubcycle=ns)
    cells = oct_cells(tree) - 1
    with runtime.Solver(tree, hp, nsubcycle=ns, uold=u) as s:
        for n in (1, 3):
            assert s.run(max_steps=n) == n
            for _ in range(n):
                orc.coarse_step()
            np.testing.assert_array_equal(s.download_state()[:, cells], orc.uold[:, cells])
            divu, enew = s.download_pressure_fix()
            np.testing.assert_array_equal(divu[cells], orc.divu[cells])
            np.testing.assert_array_equal(enew[cells], orc.enew[cells])
            assert s.t == orc.t


@pytest.mark.parametrize("pressure_fix", [False, True])
@pytest.mark.parametrize("pattern", [(2, 2), (1, 2)])
@pytest.mark.parametrize("bounds", [("outflow",) * 3, ("reflexive", None, "outflow")])
def test_finest_level_at_the_wall(cuda_lib, oracle_lib, bounds, pattern, pressure_fix):
    """A finest level with boundary octs of its own, subcycled: no alternation
    of its two buffers, and the scheduler's operations after its boundary fill.
    Levels up to 4 are complete and the steps start on level 2."""
    hp = HydroParams(gamma=1.4, riemann="hllc", slope_type=1, courant_factor=0.8, pressure_fix=pressure_fix,
                     beta_fix=0.5 if pressure_fix else 0.0)
    tree = dataclasses.replace(mesh.add_boundaries(mesh.build_tree(4), bounds), levelmin=2)
    assert all(len(tree.boundary_octs(l)[0]) > 0 for l in (2, 3, 4))
    centre = (0.05, 0.5, 0.95)

    def prim(x):
        q = np.zeros((5, len(x)))
        q[0] = 1.0 + 0.2 * np.cos(7 * x[:, 0] + 5 * x[:, 2])
        q[1], q[2], q[3] = -0.8, 0.3 * np.sin(6 * x[:, 1]), 0.7
        q[4] = np.where(((x - np.array(centre)) ** 2).sum(1) < 0.01, 20.0, 0.5)
        return q
    u = ics.fill_all_levels(tree, prim, hp.gamma)
    ns = [pattern[i % 2] for i in range(33)]
    orc = oracle.OracleRun(tree, hp, u, nsubcycle=ns)
    cells = oct_cells(tree) - 1
    with runtime.Solver(tree, hp, nsubcycle=ns, uold=u) as s:
        for n in (1, 4):
            assert s.run(max_steps=n) == n
            for _ in range(n):
                orc.coarse_step()
            np.testing.assert_array_equal(s.download_state()[:, cells], orc.uold[:, cells])
            assert s.t == orc.t
