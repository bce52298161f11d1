"""GPU: every oct is updated by one tile slot, FP64 against the oracle bit for
bit, on periodic levels with fewer octs along an axis than a tile, or not a
multiple of it: levels 1-3 of a one-cell coarse grid and of a periodic coarse
grid of three cells per axis, in the default and in every requested tile
shape, with the update read from unew (godunov_fine) and inside run()."""
import ctypes

import numpy as np
import pytest

import oracle
from ramses_b200 import mesh, runtime
from ramses_b200.params import HydroParams

pytestmark = pytest.mark.gpu


def complete_tree(n, nlevel):
    """Levels 1..nlevel complete on a periodic coarse grid of n[0] x n[1] x n[2] cells."""
    n = np.array(n)
    ncoarse = int(n.prod())
    count = [ncoarse * 8 ** l for l in range(nlevel)]
    ngm = sum(count)
    son = np.zeros(ncoarse + 8 * ngm, np.int32)
    father, nbor = np.zeros(ngm, np.int32), np.zeros((6, ngm), np.int32)
    active, coords = [np.zeros(0, np.int32)], [np.zeros((0, 3), np.int64)]
    igrid_of = None                      # of level l-1, by position
    g0 = 0
    for l in range(1, nlevel + 1):
        m = n << (l - 1)                 # octs of the level = cells of the level above
        z, y, x = np.meshgrid(*[np.arange(k) for k in m[::-1]], indexing="ij")
        c = np.stack([x.ravel(), y.ravel(), z.ravel()], 1)

        def cell(p):
            p = p % m
            if l == 1:
                return 1 + p[:, 0] + n[0] * (p[:, 1] + n[1] * p[:, 2])
            h = m >> 1
            g = igrid_of[p[:, 0] // 2 + h[0] * (p[:, 1] // 2 + h[1] * (p[:, 2] // 2))]
            return ncoarse + ((p & 1) @ np.array([1, 2, 4])) * ngm + g
        g = g0 + 1 + np.arange(len(c))
        father[g - 1] = cell(c)
        son[cell(c) - 1] = g
        for j in range(6):
            step = np.zeros(3, np.int64)
            step[j // 2] = 1 if j % 2 else -1
            nbor[j, g - 1] = cell(c + step)
        active.append(g.astype(np.int32))
        coords.append(c)
        igrid_of, g0 = g, g0 + len(c)
    return mesh.Octree(nx=int(n[0]), ny=int(n[1]), nz=int(n[2]), ncoarse=ncoarse, ngridmax=ngm, nlevelmax=nlevel,
                       levelmin=1, boxlen=1.0, son=son, father=father, nbor=nbor, active=active, coords=coords)


def state(tree, seed=3):
    rng = np.random.default_rng(seed)
    n = tree.ncell
    u = np.empty((5, n))
    u[0] = np.exp(0.4 * rng.standard_normal(n))
    u[1:4] = 0.4 * u[0] * rng.standard_normal((3, n))
    u[4] = np.exp(0.4 * rng.standard_normal(n)) / 0.4 + 0.5 * (u[1:4] ** 2).sum(0) / u[0]
    return u


def cells_of(tree, level):
    g = tree.active[level].astype(np.int64)
    return (tree.ncoarse + np.arange(8)[:, None] * tree.ngridmax + g[None, :] - 1).ravel()


@pytest.mark.parametrize("pressure_fix", [False, True])
@pytest.mark.parametrize("shape", [None, 0, 1, 2, 3, 4])
@pytest.mark.parametrize("coarse", [(1, 1, 1), (3, 3, 3), (3, 1, 5)])
def test_godunov_fine_updates_once(cuda_lib, oracle_lib, coarse, shape, pressure_fix):
    tree = complete_tree(coarse, 3)
    hp = HydroParams(gamma=1.4, riemann="hllc", slope_type=1, courant_factor=0.5, pressure_fix=pressure_fix,
                     beta_fix=0.5 if pressure_fix else 0.0)
    u = state(tree)
    for level in (1, 2, 3):
        orc = oracle.OracleRun(tree, hp, u)
        orc.set_unew(level)
        orc.godunov_fine(level, 1e-3)
        cells = cells_of(tree, level)
        with runtime.Solver(tree, hp, uold=u) as s:
            if shape is not None:
                s.set_tile_shape(level, shape)
            got = runtime_shape(s, level)
            assert all((k << (level - 1)) % (t // 2) == 0 for k, t in zip(coarse, got)), (level, got)
            s.set_unew(level)
            s.godunov_fine(level, 1e-3)
            np.testing.assert_array_equal(s.download_unew()[:, cells], orc.unew[:, cells])
            if pressure_fix:
                divu, enew = s.download_pressure_fix()
                np.testing.assert_array_equal(divu[cells], orc.divu[cells])
                np.testing.assert_array_equal(enew[cells], orc.enew[cells])


def runtime_shape(s, level):
    v = [ctypes.c_int32() for _ in range(4)]
    assert runtime.load().rb_tile_shape_info(s.tile_shape(level), *[ctypes.byref(x) for x in v]) == 0
    return [x.value for x in v[:3]]


@pytest.mark.parametrize("coarse,nlevel", [((1, 1, 1), 1), ((1, 1, 1), 2), ((3, 3, 3), 1), ((3, 3, 3), 2)])
def test_run(cuda_lib, oracle_lib, coarse, nlevel):
    tree = complete_tree(coarse, nlevel)
    hp = HydroParams(gamma=1.4, riemann="hllc", slope_type=2, courant_factor=0.5)
    u = state(tree, 5)
    orc = oracle.OracleRun(tree, hp, u)
    for _ in range(3):
        orc.coarse_step()
    with runtime.Solver(tree, hp, uold=u) as s:
        assert s.run(max_steps=3) == 3
        cells = np.concatenate([cells_of(tree, l) for l in range(1, nlevel + 1)])
        np.testing.assert_array_equal(s.download_state()[:, cells], orc.uold[:, cells])
        assert s.t == orc.t
