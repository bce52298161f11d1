"""Performance cases: the work that programs have this library do, through its
public entry points, over the range of sizes, precisions and schemes in use.

Five kinds of call:

* ``uniform``: a complete level advanced by ``Solver.uniform_run`` and read
  back for an output (the turbulent box and uniform Sedov configurations);
* ``amr``: a refined octree advanced by ``Solver.run``, coarse steps with
  subcycling, and read back (the Sedov shell and blast-clump configurations,
  with and without outflow boundaries and the pressure fix);
* ``levels``: one coarse step as a host code drives it, level routine by level
  routine, with the refinement flags of every level at its end;
* ``serve``: a batch of independent problems (uniform tubes and blasts, small
  octrees) submitted to the serving engine and drained;
* ``unsplit``: one vector sweep of the reference-layout ``unsplit`` call.

A pass advances the state it is given, so repeated passes continue the same
run, as a program does between two outputs. Inputs are seeded synthetic fields.
"""
import functools
import math

import numpy as np
import torch

from ramses_b200 import mesh, runtime, serve
from ramses_b200.params import HydroParams, RefineParams

SMALLR = 1e-10
SMALLC = 1e-10


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    def uniform(name, level, precision, riemann, slope, gamma, steps):
        return {"name": name, "kind": "uniform", "level": level, "precision": precision, "riemann": riemann,
                "slope": slope, "gamma": gamma, "steps": steps}

    def amr(name, shape, lmin, lmax, radius, outflow, precision, riemann, slope, pfix, steps):
        return {"name": name, "kind": "amr", "shape": shape, "lmin": lmin, "lmax": lmax, "radius": radius,
                "outflow": outflow, "precision": precision, "riemann": riemann, "slope": slope, "pfix": pfix,
                "steps": steps}

    return [
        # the smallest uniform run (parity and serving size): launches and latency count
        uniform("uniform_32_mixed", 5, "mixed", "hllc", 2, 1.4, 24),
        # 64^3 with the default solver and limiter of &HYDRO_PARAMS (llf, minmod), drop-in precision
        uniform("uniform_64_fp64_llf", 6, "fp64", "llf", 1, 1.4, 20),
        # an ordinary drop-in run of the turbulent box's scheme
        uniform("uniform_128_fp64", 7, "fp64", "hllc", 2, 1.001, 30),
        # the headline workload: the 256^3 turbulent box, FP32-mixed
        uniform("uniform_256_mixed", 8, "mixed", "hllc", 2, 1.001, 128),
        # Sedov on levels 6-9 inside outflow boundaries (the AMR headline)
        amr("amr_sedov_6_9_mixed", "shell", 6, 9, 0.25, True, "mixed", "hllc", 1, False, 16),
        # blast and clumps, moncen, drop-in precision
        amr("amr_clumps_6_8_fp64", "clumps", 6, 8, 0.04, False, "fp64", "hllc", 2, False, 3),
        # the dual-energy fix, which cold or high-Mach runs switch on
        amr("amr_pfix_5_8_mixed", "shell", 5, 8, 0.25, False, "mixed", "hllc", 1, True, 4),
        # a small octree with the default solver and limiter: many small launches
        amr("amr_llf_4_6_mixed", "shell", 4, 6, 0.25, False, "mixed", "llf", 1, False, 12),
        # the host code's own loop over level routines, one coarse step, with refinement flags
        {"name": "levels_5_7_fp64", "kind": "levels", "lmin": 5, "lmax": 7, "radius": 0.25, "precision": "fp64",
         "riemann": "hllc", "slope": 1, "steps": 1},
        # ensemble serving: uniform problems of two sizes and a few octrees, submitted together
        {"name": "serve_28_mixed", "kind": "serve", "dense": 24, "n_small": 32, "n_large": 64, "octrees": 4,
         "precision": "mixed", "riemann": "hllc", "slope": 1, "steps": 200},
        # one default-length vector sweep (nvector = 32) through the reference's unsplit interface
        {"name": "unsplit_32", "kind": "unsplit", "nvector": 32, "riemann": "hllc", "slope": 1, "gravity": True},
    ]


def draw(rng):
    """One more case of the same ranges (rng: random.Random)."""
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choices(["uniform", "amr", "levels", "serve", "unsplit"], [4, 4, 1, 2, 1])[0]
    precision = rng.choice(["mixed", "fp64"])
    riemann = rng.choices(["hllc", "llf", "hll"], [5, 2, 1])[0]
    slope = rng.choices([1, 2, 3], [3, 3, 1])[0]
    slow = (4 if precision == "fp64" else 1) * (2 if slope == 3 or riemann != "hllc" else 1)
    if kind == "uniform":
        level = rng.randint(4, 8)
        most = max(1, min(200, int(1.2e9 / slow / 8 ** level)))
        return {"kind": kind, "level": level, "precision": precision, "riemann": riemann, "slope": slope,
                "gamma": rng.choice([1.001, 1.4, 5.0 / 3.0]), "steps": log_int(1, most)}
    if kind == "amr":
        lmin = rng.randint(4, 6)
        lmax = min(8, lmin + rng.randint(1, 3))
        shape = rng.choice(["shell", "clumps"])
        radius = round(rng.uniform(0.15, 0.3) if shape == "shell" else rng.uniform(0.02, 0.05), 4)
        return {"kind": kind, "shape": shape, "lmin": lmin, "lmax": lmax, "radius": radius,
                "outflow": rng.random() < 0.3, "precision": precision, "riemann": riemann, "slope": slope,
                "pfix": rng.random() < 0.25, "steps": log_int(1, max(1, 24 >> (lmax - lmin)))}
    if kind == "levels":
        lmin = rng.randint(4, 6)
        return {"kind": kind, "lmin": lmin, "lmax": min(7, lmin + rng.randint(1, 2)),
                "radius": round(rng.uniform(0.15, 0.3), 4), "precision": precision, "riemann": riemann,
                "slope": slope, "steps": 1}
    if kind == "serve":
        case = {"kind": kind, "dense": log_int(2, 32), "n_small": 16 * rng.randint(1, 2),
                "n_large": 16 * rng.randint(3, 5), "octrees": rng.randint(0, 4), "precision": precision,
                "riemann": riemann, "slope": rng.choice([1, 2])}
        cells = sum(n ** 3 for n in _request_sizes(case))
        return {**case, "steps": log_int(4, max(4, min(200, int(8e8 / slow / cells))))}
    return {"kind": kind, "nvector": log_int(1, 4000), "riemann": riemann, "slope": slope,
            "gravity": rng.random() < 0.5}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _params(case):
    return HydroParams(gamma=case.get("gamma", 1.4), riemann=case["riemann"], slope_type=case["slope"],
                       courant_factor=0.8, smallr=SMALLR, smallc=SMALLC, pressure_fix=bool(case.get("pfix", False)),
                       beta_fix=0.5 if case.get("pfix") else 0.0)


CENTRE = (0.5, 0.5, 0.5)
N_CLUMPS = 12


def _clumps():
    r = np.random.default_rng(11)
    return r.uniform(0.25, 0.75, size=(N_CLUMPS, 3)), r.uniform(0.6, 1.4, size=N_CLUMPS)


@functools.lru_cache(maxsize=None)
def _uniform_tree(level):
    return mesh.uniform_tree(level)


@functools.lru_cache(maxsize=None)
def _amr_tree(shape, lmin, lmax, radius, outflow):
    """A static octree that a program would keep between two remeshes."""
    blast = mesh.sphere_refine(CENTRE, 2.5 * 0.5 ** lmax)
    if shape == "shell":
        ref = mesh.union_refine(mesh.shell_refine(CENTRE, radius, 2.5), blast)
    else:
        cen, size = _clumps()
        ref = mesh.union_refine(blast, *[mesh.sphere_refine(tuple(c), radius * s) for c, s in zip(cen, size)])
    tree = mesh.build_tree(lmin, lmax, ref)
    return mesh.add_boundaries(tree, ("outflow",) * 3) if outflow else tree


def _cells(tree):
    """[(level, cell indices from 0, integer cell coordinates)] of every cell of
    the tree by walking son from the coarse cells (cell = ncoarse +
    (ind-1)*ngridmax + igrid, ind = 1 + ix + 2 iy + 4 iz), on the GPU."""
    son = torch.from_numpy(tree.son).cuda().long()
    c = torch.arange(tree.ncoarse, device="cuda")
    xyz = torch.stack([c % tree.nx, (c // tree.nx) % tree.ny, c // (tree.nx * tree.ny)], 1)
    out = []
    for level in range(1, tree.nlevelmax + 1):
        g = son[c]
        g, xyz = g[g > 0], xyz[g > 0]
        if not len(g):
            break
        cs, xs = [], []
        for ind in range(8):
            cs.append(tree.ncoarse + ind * tree.ngridmax + g - 1)
            xs.append(2 * xyz + torch.tensor([ind & 1, (ind >> 1) & 1, ind >> 2], device="cuda"))
        c, xyz = torch.cat(cs), torch.cat(xs)
        out.append((level, c, xyz))
    return out


@functools.lru_cache(maxsize=2)
def _centres(shape, lmin, lmax, radius, outflow):
    """(cell indices, centres in the box) of every cell of an AMR tree."""
    tree = _amr_tree(shape, lmin, lmax, radius, outflow)
    off = torch.tensor(tree.offset, device="cuda", dtype=torch.float64)
    cs, xs = [], []
    for level, c, xyz in _cells(tree):
        cs.append(c)
        xs.append((xyz.double() + 0.5) * 0.5 ** level - off)
    return torch.cat(cs), torch.cat(xs)


def _cons(q, gamma):
    u = torch.empty_like(q)
    u[0] = q[0]
    for d in (1, 2, 3):
        u[d] = q[0] * q[d]
    u[4] = q[4] / (gamma - 1.0) + 0.5 * q[0] * (q[1] ** 2 + q[2] ** 2 + q[3] ** 2)
    return u


def _waves(x, seed, count, amplitude):
    """Smooth seeded field: a sum of box-periodic cosine modes at the points x [n, 3]."""
    r = np.random.default_rng(seed)
    f = torch.zeros(len(x), device="cuda", dtype=torch.float64)
    for _ in range(count):
        k = torch.tensor(2.0 * math.pi * r.integers(-3, 4, size=3), device="cuda", dtype=torch.float64)
        f += float(r.normal()) * torch.cos(x @ k + float(r.uniform(0, 2 * math.pi)))
    return amplitude * f / math.sqrt(count)


def _blast_state(x, case, seed, dx_fine):
    """Sedov-like blast in a perturbed medium (with dense clumps for that tree), conservative [5, n]."""
    r = np.random.default_rng(seed)
    q = torch.empty((5, len(x)), device="cuda", dtype=torch.float64)
    q[0] = torch.exp(_waves(x, 7 * seed + 1, 6, 0.2))
    for d in range(3):
        q[1 + d] = _waves(x, 7 * seed + 2 + d, 6, 0.1)
    q[4] = 0.05 * torch.exp(_waves(x, 7 * seed + 5, 6, 0.2))
    if case.get("shape") == "clumps":
        contrast = r.uniform(20, 100, size=N_CLUMPS)
        for c, s, k in zip(*_clumps(), contrast):
            d2 = ((x - torch.tensor(c, device="cuda")) ** 2).sum(1)
            q[0] = torch.where(d2 < (case["radius"] * s) ** 2, q[0] * float(k), q[0])
    rr = torch.sqrt(((x - 0.5) ** 2).sum(1)) / dx_fine
    inside = rr < 2.5
    energy = 10.0 ** r.uniform(-2, -1)
    q[4] = torch.where(inside, 0.4 * energy / (65.0 * dx_fine ** 3), q[4])
    return _cons(q, 1.4)


def _turbulent(n, seed, gamma):
    """Turbulent box [5, z, y, x]: log-normal density and velocities with
    steep spectra, P = 0.01 rho; Mach 5 when nearly isothermal (the box's
    own gamma 1.001), transonic otherwise."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    k = torch.fft.fftfreq(n, device="cuda", dtype=torch.float64) * n
    kk = (k[:, None, None] ** 2 + k[None, :, None] ** 2 + k[None, None, : n // 2 + 1] ** 2)
    kk[0, 0, 0] = 1.0
    amp = 1.0 / kk                       # P(k) ~ k^-4
    amp[0, 0, 0] = 0.0

    def field():
        z = torch.randn(amp.shape, device="cuda", dtype=torch.complex128, generator=g)
        f = torch.fft.irfftn(z * amp, s=(n, n, n))
        return (f - f.mean()) / f.std()
    rho = torch.exp(field())
    rho = rho / rho.mean()
    q = torch.stack([rho, field(), field(), field(), 0.01 * rho])
    cs = math.sqrt(gamma * 0.01)
    mach = 5.0 if gamma < 1.1 else 1.0
    q[1:4] *= mach * cs / math.sqrt(float((q[1:4] ** 2).sum(0).mean()))
    return _cons(q, gamma)


def _request_state(n, index, seed):
    """A serving request's [5, z, y, x]: a perturbed tube along x or a blast."""
    r = np.random.default_rng(1000 * seed + index)
    c = (torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) / n
    z, y, x = torch.meshgrid(c, c, c, indexing="ij")
    x = torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)], 1)
    if index % 2:
        return _blast_state(x, {}, 1000 * seed + index, 1.0 / n).reshape(5, n, n, n)
    q = torch.empty((5, len(x)), device="cuda", dtype=torch.float64)
    left = x[:, 0] < 0.5
    rho, p, u = 10 ** r.uniform(-1, 1, 2), 10 ** r.uniform(-2, 2, 2), r.uniform(-2, 2, 2)
    for v, pair in ((0, rho), (1, u), (4, p)):
        q[v] = torch.where(left, torch.tensor(pair[0], device="cuda"), torch.tensor(pair[1], device="cuda"))
    for d in range(3):
        w = _waves(x, 11 * (1000 * seed + index) + d, 4, 0.05)
        q[1 + d] = q[1] + w if d == 0 else w
    return _cons(q, 1.4).reshape(5, n, n, n)


def _request_sizes(case):
    """Grid sizes of the uniform requests: every third one is large."""
    return [case["n_large"] if i % 3 == 2 else case["n_small"] for i in range(case["dense"])]


def _blocks(case, seed):
    """(uin, gravin) of a vector sweep in the reference's layout, seeded."""
    nv = case["nvector"]
    r = np.random.default_rng(seed)
    q = np.empty((5, 6, 6, 6, nv))
    q[0] = np.exp(0.3 * r.standard_normal(q[0].shape))
    q[1:4] = 0.3 * r.standard_normal(q[1:4].shape)
    q[4] = np.exp(0.3 * r.standard_normal(q[0].shape))
    u = np.empty_like(q)
    u[0] = q[0]
    u[1:4] = q[0] * q[1:4]
    u[4] = q[4] / 0.4 + 0.5 * q[0] * (q[1:4] ** 2).sum(0)
    return u, (0.1 * r.standard_normal((3, 6, 6, 6, nv)) if case["gravity"] else None)


def _fortran_uniform(dense, level):
    """uold (5, ncell) of a complete grid whose finest level holds ``dense``
    [5, z, y, x] and whose coarser levels hold its means."""
    tree = _uniform_tree(level)
    grids = {level: dense}
    for l in range(level - 1, 0, -1):
        n = 2 ** l
        grids[l] = grids[l + 1].reshape(5, n, 2, n, 2, n, 2).mean((2, 4, 6))
    u = torch.zeros((5, tree.ncell), device="cuda", dtype=torch.float64)
    for l, c, xyz in _cells(tree):
        n = 2 ** l
        u[:, c] = grids[l].reshape(5, -1)[:, xyz[:, 0] + n * (xyz[:, 1] + n * xyz[:, 2])]
    return u


def _host(t):
    """A tensor's values in pinned host memory, where a program that exchanges state with a GPU keeps them."""
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def _amr_host_state(case, seed, shape, outflow):
    key = (shape, case["lmin"], case["lmax"], case["radius"], outflow)
    tree = _amr_tree(*key)
    c, x = _centres(*key)
    u = torch.zeros((5, tree.ncell), device="cuda", dtype=torch.float64)
    u[0], u[4] = 1.0, 1.0                # unused slots
    u[:, c] = _blast_state(x, case, seed, 0.5 ** case["lmax"])
    return tree, _host(u)


def prepare(case, seed):
    hp = _params(case)
    if case["kind"] == "unsplit":
        uin, grav = _blocks(case, seed)
        return {"case": case, "hp": hp, "uin": uin, "grav": grav}
    if case["kind"] == "serve":
        dense = [_host(_request_state(n, i, seed)) for i, n in enumerate(_request_sizes(case))]
        octrees = []
        for i in range(case["octrees"]):
            sub = {"lmin": 5, "lmax": 6, "radius": 0.25 - 0.02 * i}
            octrees.append(_amr_host_state(sub, 100 * seed + i, "shell", False))
        return {"case": case, "server": serve.Server(hp, precision=case["precision"]), "dense": dense,
                "octrees": octrees}
    if case["kind"] == "uniform":
        tree = _uniform_tree(case["level"])
        u = _host(_fortran_uniform(_turbulent(2 ** case["level"], seed, case["gamma"]), case["level"]))
    else:
        tree, u = _amr_host_state(case, seed, case.get("shape", "shell"), bool(case.get("outflow", False)))
    solver = runtime.Solver(tree, hp, precision=case["precision"], uold=u)
    state = {"case": case, "solver": solver, "out": u}     # u: the host's copy of uold from here on
    if case["kind"] == "levels":
        state["flags"] = np.zeros(tree.ncell + 1, np.int32)
        state["refine"] = RefineParams(err_grad_d=0.1, err_grad_p=0.1)
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _level_step(s, tree, level, dt_above):
    """amr_step's hydro calls of one level, with subcycling, as a host code issues them."""
    dt = s.courant_fine(level)[0]
    if dt_above is not None:
        dt = min(dt, dt_above / 2.0)
    s.set_unew(level)
    if level < tree.nlevelmax and tree.noct(level + 1):
        dt = _level_step(s, tree, level + 1, dt) + _level_step(s, tree, level + 1, dt)
    s.godunov_fine(level, dt)
    s.set_uold(level)
    s.upload_fine(level)
    return dt


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "unsplit":
        return runtime.unsplit(state["hp"], state["uin"], state["grav"], 1.0 / 64, 2e-3)
    if kind == "serve":
        srv = state["server"]
        ids = [srv.submit_dense(u, max_steps=case["steps"], outflow_mask=0 if i % 2 else 1)
               for i, u in enumerate(state["dense"])]
        ids += [srv.submit_octree(t, u, max_steps=max(1, case["steps"] // 8)) for t, u in state["octrees"]]
        srv.drain()
        return [srv.results.pop(i) for i in ids]
    s = state["solver"]
    if kind == "uniform":
        s.uniform_run(case["steps"])
    elif kind == "amr":
        s.run(max_steps=case["steps"])
    else:
        tree = s.tree
        flags = state["flags"]
        flags[:] = 0
        for _ in range(case["steps"]):
            _level_step(s, tree, tree.levelmin, None)
        for l in range(tree.levelmin - 1, 0, -1):
            s.upload_fine(l)
        for l in range(tree.levelmin, tree.nlevelmax):
            s.hydro_flag(l, state["refine"], flags)
        u = s.download_state(state["out"])
        return [u[0], u[1], u[2], u[3], u[4], flags]
    u = s.download_state(state["out"])
    return [u[0], u[1], u[2], u[3], u[4]]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
#: floating-point operations of one cell update (slopes, trace, three Riemann problems, update, wave speed)
FLOPS = {"hllc": 784, "hll": 760, "llf": 730}


def _leaf_updates(tree, steps):
    def of(level):
        n = tree.leaf_cells(level)
        return n + 2 * of(level + 1) if level < tree.nlevelmax and tree.noct(level + 1) else n
    return steps * of(tree.levelmin)


def work(case):
    """80 bytes for each leaf-cell update (five FP64 values read, five
    written) and the state that the pass returns, read once for it."""
    f = FLOPS[case["riemann"]]
    if case["kind"] == "unsplit":
        # 6^3 cells in (states, gravity), 36 faces of 7 values out; 32 traced cells and 36 faces of arithmetic
        n = case["nvector"]
        return {"bytes": n * 8.0 * (216 * (8 if case["gravity"] else 5) + 36 * 7), "flops": n * 12.0 * f}
    if case["kind"] == "serve":
        cells = sum(n ** 3 for n in _request_sizes(case))
        updates, size = cells * case["steps"], 40.0 * cells
        for i in range(case["octrees"]):
            t = _amr_tree("shell", 5, 6, 0.25 - 0.02 * i, False)
            updates += _leaf_updates(t, max(1, case["steps"] // 8))
            size += 40.0 * t.ncell
        return {"bytes": 80.0 * updates + size, "flops": float(f) * updates}
    if case["kind"] == "uniform":
        n = 8 ** case["level"]
        return {"bytes": 80.0 * n * case["steps"] + 40.0 * n, "flops": float(f) * n * case["steps"]}
    t = _amr_tree(case.get("shape", "shell"), case["lmin"], case["lmax"], case["radius"],
                  bool(case.get("outflow", False)))
    updates = _leaf_updates(t, case["steps"])
    return {"bytes": 80.0 * updates + 40.0 * sum(8 * t.noct(l) for l in range(1, t.nlevelmax + 1)),
            "flops": float(f) * updates}


def tolerance(case):
    """The FP64 path keeps the reference's order of operations, bit for bit.
    FP32-mixed: slopes, trace and fluxes round at 6e-8; the figures are about
    four times what the path differs by from 64-bit arithmetic over three
    passes of a case. Shocks amplify a rounding, most in a few cells of the
    turbulent box; a transverse momentum near zero shows it most in a tube."""
    if case["kind"] == "unsplit" or case["precision"] == "fp64":
        return "exact"
    return {"uniform": {"rel": 2e-6, "max": 6e-4}, "serve": {"rel": 6e-6, "max": 2e-4}}.get(
        case["kind"], {"rel": 8e-7, "max": 3e-5})


# ---------------------------------------------------------------------------
# the same in 64 bits, plain torch
# ---------------------------------------------------------------------------
def _slopes(q, slope, dims):
    """Limited slopes [direction][5, ...] of uslope, directions x, y, z."""
    out = []
    if slope == 3:
        lo = torch.full_like(q, math.inf)
        hi = torch.full_like(q, -math.inf)
        for i in (-1, 0, 1):
            for j in (-1, 0, 1):
                for k in (-1, 0, 1):
                    d = torch.roll(q, (i, j, k), dims) - q
                    lo, hi = torch.minimum(lo, d), torch.maximum(hi, d)
        dc = [0.5 * (torch.roll(q, -1, d) - torch.roll(q, 1, d)) for d in dims]
        dff = 0.5 * (dc[0].abs() + dc[1].abs() + dc[2].abs())
        lim = torch.minimum(lo.abs(), hi.abs()) / torch.where(dff > 0, dff, torch.ones_like(dff))
        lim = torch.where(dff > 0, lim.clamp(max=1.0), torch.ones_like(lim))
        return [lim * d for d in dc]
    for d in dims:
        a, b = q - torch.roll(q, 1, d), torch.roll(q, -1, d) - q
        m = torch.minimum(a.abs(), b.abs())
        if slope == 1:
            s = torch.sign(a) * m
        else:
            c = 0.5 * (a + b)
            s = torch.sign(c) * torch.minimum(2.0 * m, c.abs())
        out.append(torch.where(a * b <= 0, torch.zeros_like(s), s))
    return out


def _riemann(kind, ql, qr, gamma):
    """Fluxes (mass, normal momentum, energy, two transverse momenta, thermal
    energy) of states (rho, u_n, P, u_t1, u_t2)."""
    smallp = SMALLC ** 2 / gamma
    rl, rr = ql[0].clamp(min=SMALLR), qr[0].clamp(min=SMALLR)
    pl, pr = torch.maximum(ql[2], rl * smallp), torch.maximum(qr[2], rr * smallp)
    ul, ur = ql[1], qr[1]
    ent = 1.0 / (gamma - 1.0)
    if kind == "hllc":
        el, er = pl * ent, pr * ent
        tl = el + 0.5 * rl * (ul ** 2 + ql[3] ** 2 + ql[4] ** 2)
        tr = er + 0.5 * rr * (ur ** 2 + qr[3] ** 2 + qr[4] ** 2)
        c = torch.maximum((gamma * pl / rl).clamp(min=SMALLC ** 2).sqrt(), (gamma * pr / rr).clamp(min=SMALLC ** 2).sqrt())
        sl, sr = torch.minimum(ul, ur) - c, torch.maximum(ul, ur) + c
        cl, cr = rl * (ul - sl), rr * (sr - ur)
        us = (cr * ur + cl * ul + (pl - pr)) / (cr + cl)
        ps = (cr * pl + cl * pr + cl * cr * (ul - ur)) / (cr + cl)
        lft, out_l = us > 0, sl > 0
        star = ~out_l & (lft | (sr > 0))
        side = out_l | lft
        pick = lambda a, b: torch.where(side, a, b)  # noqa: E731
        r0, u0, s0, p0, t0, e0 = pick(rl, rr), pick(ul, ur), pick(sl, sr), pick(pl, pr), pick(tl, tr), pick(el, er)
        k = (s0 - u0) / (s0 - us)
        r = torch.where(star, r0 * k, r0)
        u = torch.where(star, us, u0)
        p = torch.where(star, ps, p0)
        t = torch.where(star, ((s0 - u0) * t0 - p0 * u0 + ps * us) / (s0 - us), t0)
        e = torch.where(star, e0 * k, e0)
        m = r * u
        return [m, m * u + p, (t + p) * u, m * torch.where(lft, ql[3], qr[3]), m * torch.where(lft, ql[4], qr[4]), u * e]
    cl, cr = (gamma * pl / rl).sqrt(), (gamma * pr / rr).sqrt()
    cons, flux = [], []
    for q in (ql, qr):
        e = q[2] * ent + 0.5 * q[0] * (q[1] ** 2 + q[3] ** 2 + q[4] ** 2)
        u = [q[0], q[0] * q[1], e, q[0] * q[3], q[0] * q[4], q[2] * ent]
        cons.append(u)
        flux.append([u[1], u[1] * q[1] + q[2], q[1] * (e + q[2])] + [q[1] * w for w in u[3:]])
    if kind == "llf":
        c = torch.maximum(ul.abs() + cl, ur.abs() + cr)
        return [0.5 * (a + b - c * (w - v)) for a, b, v, w in zip(*flux, *cons)]
    sl = (torch.minimum(ul, ur) - torch.maximum(cl, cr)).clamp(max=0)
    sr = (torch.maximum(ul, ur) + torch.maximum(cl, cr)).clamp(min=0)
    return [(sr * a - sl * b + sr * sl * (w - v)) / (sr - sl) for a, b, v, w in zip(*flux, *cons)]


def _prim(u, gamma):
    r = u[0].clamp(min=SMALLR)
    v = u[1:4] / r
    e = (u[4] / r - 0.5 * (v ** 2).sum(0)).clamp(min=SMALLC ** 2 / gamma / (gamma - 1.0))
    return torch.stack([r, v[0], v[1], v[2], (gamma - 1.0) * r * e])


def _fluxes(u, dtdx, half_dt_g, kind, slope, gamma):
    """[direction] -> (flux of rho, mx, my, mz, E; velocity average; thermal
    flux) through each cell's lower face; u [5, z, y, x, ...]."""
    q = _prim(u, gamma)
    if half_dt_g is not None:
        q[1:4] += half_dt_g
    dims = (3, 2, 1)
    dq = _slopes(q, slope, dims)
    r, p = q[0], q[4]
    div = dq[0][1] + dq[1][2] + dq[2][3]
    adv = q[1] * dq[0] + q[2] * dq[1] + q[3] * dq[2]
    src = -adv
    src[0] -= div * r
    src[4] -= div * gamma * p
    for d in range(3):
        src[1 + d] -= dq[d][4] / r
    mid = q + 0.5 * dtdx * src
    del src, adv
    out = []
    for d in range(3):
        lo, hi = mid - 0.5 * dq[d], mid + 0.5 * dq[d]
        lo[0] = torch.where(lo[0] < SMALLR, r, lo[0])
        hi[0] = torch.where(hi[0] < SMALLR, r, hi[0])
        left = torch.roll(hi, 1, dims[d])
        order = [0, 1 + d, 4] + [1 + e for e in range(3) if e != d]
        f = _riemann(kind, [left[i] for i in order], [lo[i] for i in order], gamma)
        g = [None] * 5
        for i, x in zip(order, f):
            g[i] = x
        g[order[2]] = f[2]
        out.append((torch.stack(g), 0.5 * (left[1 + d] + lo[1 + d]), f[5]))
    return out


def _grow(u, outflow):
    """Two ghost cells on each side: the periodic image, or the edge cell where bit d of outflow is set."""
    for d, dim in ((0, 3), (1, 2), (2, 1)):
        n = u.shape[dim]
        at = torch.arange(-2, n + 2, device=u.device)
        at = at.clamp(0, n - 1) if outflow & (1 << d) else at % n
        u = u.index_select(dim, at)
    return u


def _advance(u, steps, kind, slope, gamma, outflow=0, courant=0.8):
    n = u.shape[1]
    dx = 1.0 / n
    for _ in range(steps):
        r = u[0].clamp(min=SMALLR)
        v = u[1:4] / r
        p = torch.maximum((gamma - 1.0) * (u[4] - 0.5 * r * (v ** 2).sum(0)), r * SMALLC ** 2 / gamma)
        speed = float((3.0 * (gamma * p / r).sqrt() + v.abs().sum(0)).max())
        dt = min(1.0 / SMALLC, courant * dx / SMALLC, dx / speed * (math.sqrt(1.0 + 2e-4 * courant) - 1.0) / 1e-4)
        f = _fluxes(_grow(u, outflow), dt / dx, None, kind, slope, gamma)
        c = slice(2, 2 + n)
        for (flux, _, _), dim in zip(f, (3, 2, 1)):
            diff = flux - torch.roll(flux, -1, dim)
            u = u + dt / dx * diff[:, c, c, c]
        del f
    return u


def exact(case, seed):
    kind, slope = case["riemann"], case["slope"]
    if case["kind"] == "unsplit":
        uin, grav = _blocks(case, seed)
        dx, dt = 1.0 / 64, 2e-3
        g = None if grav is None else 0.5 * dt * torch.from_numpy(grav).cuda()
        f = _fluxes(torch.from_numpy(uin).cuda(), dt / dx, g, kind, slope, 1.4)
        nv = case["nvector"]
        flux = torch.zeros((3, 5, 3, 3, 3, nv), dtype=torch.float64)
        tmp = torch.zeros((3, 2, 3, 3, 3, nv), dtype=torch.float64)
        for d in range(3):
            ext = [2, 2, 2]              # faces 1..3 along the direction, cells 1..2 across
            ext[2 - d] = 3
            at = tuple(slice(2, 2 + e) for e in ext)
            to = tuple(slice(0, e) for e in ext)
            flux[(d, slice(None)) + to] = (f[d][0] * dt / dx)[(slice(None),) + at].cpu()
            tmp[(d, 0) + to] = (f[d][1] * dt / dx)[at].cpu()
            tmp[(d, 1) + to] = (f[d][2] * dt / dx)[at].cpu()
        return flux, tmp
    if case["kind"] == "uniform":
        n = 2 ** case["level"]
        u = _advance(_turbulent(n, seed, case["gamma"]), case["steps"], kind, slope, case["gamma"])
        u = _fortran_uniform(u, case["level"])
        return [x.cpu() for x in u]
    if case["kind"] == "serve":
        got = []
        for i, n in enumerate(_request_sizes(case)):
            got.append(_advance(_request_state(n, i, seed), case["steps"], kind, slope, 1.4, 0 if i % 2 else 1).cpu())
        return got + [None] * case["octrees"]
    return None                          # octrees in plain tensors take minutes
