"""GPU: the run-time scheme variant of the oct-tile kernel (slope types 0, 3,
7 and 8, the acoustic and exact solvers, difmag, PLMDE with llf and hll) in
every tile shape: FP64 equals the oracle bit for bit (the exact solver, which
calls pow, within its rounding) with and without the pressure fix, FP32-mixed
gives the same bits in every shape; and its default shapes at the sizes where
the rule changes."""
import numpy as np
import pytest

import oracle
from ramses_b200 import runtime

from helpers import oct_cells, sedov_amr, sedov_uniform

pytestmark = pytest.mark.gpu

SCHEMES = [dict(slope_type=3, riemann="hllc"), dict(slope_type=3, riemann="llf", scheme="plmde"),
           dict(slope_type=0, riemann="hll"), dict(slope_type=7, riemann="llf"), dict(slope_type=8, riemann="hllc"),
           dict(slope_type=1, riemann="acoustic"), dict(slope_type=2, riemann="exact"),
           dict(slope_type=1, riemann="hllc", difmag=0.2), dict(slope_type=2, riemann="hll", scheme="plmde")]


def problem(levels, scheme, pressure_fix):
    tree, hp, u = sedov_amr(*levels)
    for k, v in scheme.items():
        setattr(hp, k, v)
    hp.pressure_fix, hp.beta_fix = pressure_fix, 0.5 if pressure_fix else 0.0
    u = u.copy()
    rng = np.random.default_rng(5)
    u[0] *= 1.0 + 0.2 * rng.random(u.shape[1])
    u[1:4] += 0.1 * u[0] * (rng.random((3, u.shape[1])) - 0.5)
    u[4] += 0.5 * (u[1:4] ** 2).sum(0) / np.maximum(u[0], 1e-10) + 0.05
    return tree, hp, u


def run(tree, hp, u, precision, shape):
    with runtime.Solver(tree, hp, precision=precision, uold=u) as s:
        if shape is not None:
            for l in range(tree.levelmin, tree.nlevelmax + 1):
                s.set_tile_shape(l, shape)
        assert s.run(max_steps=2) == 2
        out = [s.download_state()]
        return out + list(s.download_pressure_fix()) if hp.pressure_fix else out


@pytest.mark.parametrize("pressure_fix", [False, True])
@pytest.mark.parametrize("scheme", SCHEMES, ids=lambda s: "-".join(str(v) for v in s.values()))
@pytest.mark.parametrize("levels", [(3, 5)])
def test_shapes(cuda_lib, oracle_lib, levels, scheme, pressure_fix):
    tree, hp, u = problem(levels, scheme, pressure_fix)
    orc = oracle.OracleRun(tree, hp, u)
    for _ in range(2):
        orc.coarse_step()
    cells = oct_cells(tree) - 1
    ref = [orc.uold, orc.divu, orc.enew][:3 if pressure_fix else 1]
    if hp.riemann == "exact":
        # pow on the device and on the host differ by an ulp or two: some 1e-15
        # per face, a hundred faces per cell in two coarse steps
        out = run(tree, hp, u, "fp64", None)
        for a, b in zip(ref, out):
            a, b = a[..., cells], b[..., cells]
            assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(a)
        ref = out
    first = None
    for shape in (None, 0, 1, 2, 3, 4):
        for a, b in zip(ref, run(tree, hp, u, "fp64", shape)):
            np.testing.assert_array_equal(a[..., cells], b[..., cells], err_msg=str(shape))
        mixed = run(tree, hp, u, "mixed", shape)
        first = first or mixed
        for a, b in zip(first, mixed):
            np.testing.assert_array_equal(a[..., cells], b[..., cells], err_msg="mixed %s" % shape)


@pytest.mark.parametrize("precision,level,shape", [("fp64", 3, 0), ("fp64", 4, 0), ("fp64", 5, 3), ("fp64", 6, 4),
                                                   ("mixed", 4, 0), ("mixed", 5, 2), ("mixed", 6, 3)])
def test_default_shape(cuda_lib, precision, level, shape):
    tree, hp, u = sedov_uniform(level, slope_type=3)
    with runtime.Solver(tree, hp, precision=precision, uold=u) as s:
        assert s.tile_shape(level) == shape
        assert s.tile_shape(1) == 0          # one oct: no wider tile
    hp.slope_type = 1                        # a compiled variant
    with runtime.Solver(tree, hp, precision=precision, uold=u) as s:
        assert s.tile_shape(level) == (4 if precision == "fp64" and level == 6 else 3)
