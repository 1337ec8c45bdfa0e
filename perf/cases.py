"""What this framework is used for, as measurable cases.

Every case is the call pattern of a replacement ``solver::solve``: the state goes in from host
memory (``lee_upload_state``), the RK loop runs (``lee_advance``, ``lee_advance_blocks``, the
FIX_CFL loop or ``lee_adjoint_gradient``) and the result comes back to host memory. Host buffers
are pinned and kept, as a program with its own time loop keeps them. The FP32-compensated form
hands its results on in single precision, as single-precision PLOT3D solution files hold them.

Kinds (``case["kind"]``):

* ``cfl_loop``  a small block stepped by the FIX_CFL loop: CFL, rescaled dt and one step per call,
                then the report's minima and maxima.
* ``pulse2d``   2-D Cartesian block, uniform mean, sponges (Gaussian pulses).
* ``curvi3d``   3-D curvilinear block, uniform mean flow, sponges (Gaussian pulses).
* ``wall3d``    3-D curvilinear block with a slip wall, a Neumann face and a sheared mean flow.
* ``cylinder``  Cartesian background and O-grid around a cylinder, overset, shear layer, monopole.
* ``batch``     many independent 2-D instances with their own sizes, sources and time steps.
* ``adjoint``   gradient of a microphone objective with respect to a distributed source.

``exact`` is the same scheme in plain torch, FP64: every difference and filter is a dense matrix
per grid line direction.
"""
import math

import numpy as np
import torch

from camille_b200 import api
from camille_b200 import cases as builders

GAMMA = 1.4
DEVICE = "cuda"
_LIB = []


def listed():
    return [
        # the smallest call: a deck in FIX_CFL mode steps one step per call, 64 x 48 points
        {"name": "cfl_loop_64x48_f64", "kind": "cfl_loop", "nx": 64, "ny": 48, "nz": 1, "prec": "f64", "steps": 8},
        # the plain FP64 2-D configuration: 256^2, 20-cell sponges
        {"name": "pulse2d_256_f64", "kind": "pulse2d", "nx": 256, "ny": 256, "nz": 1, "prec": "f64", "steps": 200},
        # an odd-sized 2-D block (2^k + 1 points in one direction), compensated
        {"name": "pulse2d_513x385_f32", "kind": "pulse2d", "nx": 513, "ny": 385, "nz": 1, "prec": "f32",
         "steps": 100},
        # the headline: 256^3 curvilinear, Mach 0.5, compensated
        {"name": "curvi3d_256_f32", "kind": "curvi3d", "nx": 256, "ny": 256, "nz": 256, "prec": "f32",
         "steps": 100},
        # the same in plain FP64 on a block with unequal sides
        {"name": "curvi3d_160x144x128_f64", "kind": "curvi3d", "nx": 160, "ny": 144, "nz": 128, "prec": "f64",
         "steps": 60},
        # a 3-D grid of odd sides, as 2^k + 1 grids and cut blocks have them
        {"name": "curvi3d_129x113x97_f32", "kind": "curvi3d", "nx": 129, "ny": 113, "nz": 97, "prec": "f32",
         "steps": 60},
        # the 11-point optimised difference and filter (FDO11P, SFO11P)
        {"name": "curvi3d_96_fdo11_f64", "kind": "curvi3d", "nx": 96, "ny": 96, "nz": 96, "prec": "f64",
         "steps": 40, "scheme": "FDO11P"},
        # sheared mean over a slip wall: mean gradients, BC lines
        {"name": "wall3d_128x112x96_f32", "kind": "wall3d", "nx": 128, "ny": 112, "nz": 96, "prec": "f32",
         "steps": 60},
        # the overset configuration: 512^2 background, 384 x 96 O-grid
        {"name": "cylinder_512_f32", "kind": "cylinder", "nx": 512, "ny": 384, "nz": 96, "prec": "f32",
         "steps": 100},
        # the batched configuration: 64 instances, sides 64 to 512
        {"name": "batch_64_f32", "kind": "batch", "nx": 64, "ny": 512, "nz": 64, "prec": "f32", "steps": 60},
        # a smaller batch in plain FP64
        {"name": "batch_24_f64", "kind": "batch", "nx": 64, "ny": 300, "nz": 24, "prec": "f64", "steps": 60},
        # the adjoint gradient, checkpoints with recomputed segments
        {"name": "adjoint_128_f32", "kind": "adjoint", "nx": 128, "ny": 128, "nz": 128, "prec": "f32",
         "steps": 80},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cfl_loop", "pulse2d", "pulse2d", "curvi3d", "curvi3d", "curvi3d", "wall3d", "cylinder",
                       "batch", "adjoint"])
    prec = rng.choice(["f64", "f32"])
    c = {"kind": kind, "prec": prec}
    if kind == "cfl_loop":
        c.update(nx=_log_int(rng, 32, 128), ny=_log_int(rng, 32, 128), nz=1, steps=rng.randint(4, 12))
    elif kind == "pulse2d":
        c.update(nx=_log_int(rng, 64, 640), ny=_log_int(rng, 64, 640), nz=1, steps=rng.randint(60, 200))
    elif kind == "curvi3d":
        s = [_log_int(rng, 32, 200) for _ in range(3)]
        c.update(nx=s[0], ny=s[1], nz=s[2], steps=rng.randint(30, 60))
        if rng.random() < 0.25:
            c["scheme"] = "FDO11P"
    elif kind == "wall3d":
        s = [_log_int(rng, 32, 144) for _ in range(3)]
        c.update(nx=s[0], ny=s[1], nz=s[2], steps=rng.randint(30, 60))
    elif kind == "cylinder":
        nb = _log_int(rng, 192, 576)
        c.update(nx=nb, ny=int(nb * rng.uniform(0.65, 0.85)), nz=_log_int(rng, 64, 112), steps=rng.randint(50, 120))
    elif kind == "batch":
        lo = rng.randint(48, 96)
        c.update(nx=lo, ny=rng.randint(128, 480), nz=rng.randint(8, 56), steps=rng.randint(30, 80))
    else:
        n = _log_int(rng, 64, 144)
        c.update(nx=n, ny=n, nz=n, steps=rng.randint(40, 80))
    return c


# ---- inputs ---------------------------------------------------------------------------------

def _pulses(rng, dims, halfwidth, count=8, amplitude=1e-3, slots=5):
    """Smooth perturbations of every slot: ``count`` Gaussian pulses in index space, away from the
    edges, with a random amplitude per slot (w' is zero in 2-D)."""
    nx, ny, nz = dims
    g = []
    for n in dims:
        c = rng.uniform(0.25 * (n - 1), 0.75 * (n - 1), size=count) if n > 1 else np.zeros(count)
        g.append(np.exp(-math.log(2.0) * ((np.arange(n) - c[:, None]) / halfwidth) ** 2))
    zy = (g[2][:, :, None] * g[1][:, None, :]).reshape(count, nz * ny)
    out = np.zeros((5, nz, ny, nx))
    for v in range(slots):
        if v == 3 and nz == 1:
            continue
        a = amplitude * rng.normal(size=count)
        np.matmul((a[:, None] * zy).T, g[0], out=out[v].reshape(nz * ny, nx))
    return out


def _grid3d(nx, ny, nz, amp=0.1):
    """x = xi + amp sin(2 pi eta / Ny) sin(2 pi zeta / Nz) and its cyclic permutations."""
    c = [np.arange(n, dtype=np.float64) for n in (nx, ny, nz)]
    s = [np.sin(2.0 * math.pi * c[d] / n) for d, n in enumerate((nx, ny, nz))]
    x = c[0][None, None, :] + amp * (s[2][:, None, None] * s[1][None, :, None])
    y = c[1][None, :, None] + amp * (s[2][:, None, None] * s[0][None, None, :])
    z = c[2][:, None, None] + amp * (s[1][None, :, None] * s[0][None, None, :])
    return x, y, z


def _sponges(dims, width, constant, skip=()):
    """Freund ambient zones on every side, the strengths C (depth / width)^2 given by the caller."""
    num_dim = 2 if dims[2] == 1 else 3
    out = []
    for bd in builders.sponge_frame(num_dim, dims, width):
        if (bd.dir, bd.end) in skip:
            continue
        shape = [bd.hi[d] - bd.lo[d] + 1 for d in (2, 1, 0)]
        k = np.arange(width, dtype=np.float64)
        depth = (width - 1 - k) if bd.end == 0 else k
        ax = [1, 1, 1]
        ax[2 - bd.dir] = width
        prof = (constant * (depth / (width - 1)) ** 2).reshape(ax)
        bd.sigma = np.ascontiguousarray(np.broadcast_to(prof, shape))
        out.append(bd)
    return out


def _uniform_mean(shape, velocity):
    mean = np.zeros((5,) + shape)
    for q in range(3):
        if velocity[q]:
            mean[1 + q] = velocity[q]
    mean[4] = 1.0 / GAMMA
    return mean


def _problem(case, seed):
    """The inputs of a case as a builders.Case: grids, means, boundaries, sources and states."""
    rng = np.random.default_rng([seed, 77])
    kind, nx, ny, nz = case["kind"], case["nx"], case["ny"], case["nz"]
    if kind in ("cfl_loop", "pulse2d"):
        dx = 100.0 / 255.0
        x = np.ascontiguousarray(np.broadcast_to((np.arange(nx) * dx)[None, None, :], (1, ny, nx)))
        y = np.ascontiguousarray(np.broadcast_to((np.arange(ny) * dx)[None, :, None], (1, ny, nx)))
        blk = builders.Block(x, y, np.zeros_like(x), _uniform_mean(x.shape, (0.0, 0.0, 0.0)),
                             _pulses(rng, (nx, ny, 1), 3.0))
        width = max(4, round(20 * min(nx, ny) / 256))
        return builders.Case(name=kind, num_dim=2, blocks=[blk], sponge_constant=5.0,
                             boundaries=_sponges(blk.dims, width, 5.0))
    if kind == "curvi3d":
        x, y, z = _grid3d(nx, ny, nz)
        blk = builders.Block(x, y, z, _uniform_mean(x.shape, (0.5, 0.0, 0.0)), _pulses(rng, (nx, ny, nz), 4.0))
        c = builders.Case(name=kind, num_dim=3, blocks=[blk], sponge_constant=1.0,
                          boundaries=_sponges(blk.dims, max(4, round(min(nx, ny, nz) / 16)), 1.0))
        if case.get("scheme") == "FDO11P":
            c.fd_scheme, c.filter_scheme = "FDO11P", "SFO11P"
        return c
    if kind == "wall3d":
        x, y, z = _grid3d(nx, ny, nz)
        mean = _uniform_mean(x.shape, (0.0, 0.0, 0.0))
        mean[0] = 0.05 * np.tanh((z - 0.5 * nz) / 6.0)
        mean[1] = 0.3 * (1.0 + 0.5 * np.tanh((z - 0.5 * nz) / 6.0))
        blk = builders.Block(x, y, z, mean, _pulses(rng, (nx, ny, nz), 4.0))
        m = (nx - 1, ny - 1, nz - 1)
        bnd = [builders.Boundary(0, "wall_slip_kinematic", 2, 0, (0, 0, 0), (m[0], m[1], 0)),
               builders.Boundary(0, "neumann", 0, 1, (m[0], 0, 0), m)]
        bnd += _sponges(blk.dims, max(4, round(min(nx, ny, nz) / 12)), 1.0, skip=((2, 0), (0, 1)))
        return builders.Case(name=kind, num_dim=3, blocks=[blk], sponge_constant=1.0, boundaries=bnd)
    if kind == "cylinder":
        a = rng.uniform(0.0, 2.0 * math.pi)
        return builders.cylinder2d(nb=nx, ntheta=ny, nr=nz, first_cell=0.005 * 96 / nz,
                                   length=80.0 * nx / 512, amplitude=1e-3 * rng.uniform(0.5, 1.5),
                                   source=(2.0, rng.uniform(-0.5, 0.5)),
                                   pulse=(3.0 * math.cos(a), 3.0 * math.sin(a), 1e-3, rng.uniform(0.4, 0.6)))
    if kind == "batch":
        # the sizes belong to the case (the same for every seed), the instances' data to the seed
        sides = np.random.default_rng([nx, ny, nz]).uniform(math.log(nx), math.log(ny), size=nz)
        sides = np.rint(np.exp(sides)).astype(int)
        blocks, bnd = [], []
        dx = 100.0 / 255.0
        for b, n in enumerate(int(s) for s in sides):
            c1 = dx * (np.arange(n) - 0.5 * (n - 1))
            yy, xx = np.meshgrid(c1, c1, indexing="ij")
            om = rng.uniform(math.pi / 10.0, math.pi / 3.0)
            pos = rng.uniform(-0.25, 0.25, size=2) * (n - 1) * dx
            blocks.append(builders.Block(xx[None].copy(), yy[None].copy(), np.zeros((1, n, n)),
                                         _uniform_mean((1, n, n), (rng.uniform(0.0, 0.6), 0.0, 0.0)),
                                         _pulses(rng, (n, n, 1), 3.0, count=2),
                                         monopole=(pos[0], pos[1], 0.0, 1e-3, om, 3.0 * dx, 2.0 * math.pi / om)))
            for bd in _sponges((n, n, 1), max(4, round(20 * n / 256)), 5.0):
                bd.block = b
                bnd.append(bd)
        return builders.Case(name=kind, num_dim=2, blocks=blocks, sponge_constant=5.0, boundaries=bnd)
    # adjoint: a distributed source of 16^3 amplitudes around the centre, 64 microphones on an arc
    n = nx
    x, y, z = _grid3d(n, n, n)
    blk = builders.Block(x, y, z, _uniform_mean(x.shape, (0.5, 0.0, 0.0)), _pulses(rng, (n, n, n), 4.0))
    h = 4.0 * n / 192.0
    o = 0.5 * (n - 1) - 7.5 * h
    src = builders.DistributedSource(0, 0.4 * math.pi, (o, o, o), (h, h, h),
                                     rng.normal(0.0, 1e-3, size=(16, 16, 16)))
    th = np.linspace(-0.5 * math.pi, 0.5 * math.pi, 64)
    ii = np.rint(0.5 * (n - 1) + 0.28 * n * np.cos(th)).astype(np.int64)
    jj = np.rint(0.5 * (n - 1) + 0.28 * n * np.sin(th)).astype(np.int64)
    mic = np.unique(ii + n * (jj + n * (n // 2)))
    return builders.Case(name=kind, num_dim=3, blocks=[blk], sponge_constant=1.0, distributed=src,
                         microphones=builders.Microphones(0, mic, 1.0),
                         boundaries=_sponges(blk.dims, max(4, round(n / 16)), 1.0))


def _time_steps(case, prob):
    """FIX_DT time steps of the blocks: RK4 at about CFL 0.5 of the sound speed plus the mean flow."""
    if case["kind"] == "batch":
        return [0.2 / (1.0 + float(b.mean[1, 0, 0, 0])) for b in prob.blocks]
    if case["kind"] == "pulse2d":
        return [0.13]
    if case["kind"] == "cylinder":
        # the first cell at the wall sets it
        return [0.5 * 0.005 * 96 / case["nz"]]
    return [0.28]


# ---- the measured calls ---------------------------------------------------------------------

def prepare(case, seed):
    if not _LIB:
        _LIB.append(api.product_library())
    prob = _problem(case, seed)
    prec = api.FP32_COMPENSATED if case["prec"] == "f32" else api.FP64
    solver = api.Solver(_LIB[0], prob, precision=prec, upload=False)
    n = sum(b.npoints for b in prob.blocks)
    h_in = torch.empty(5 * n, dtype=torch.float64, pin_memory=True)
    h_out = torch.zeros(5 * n, dtype=torch.float64, pin_memory=True)
    ins, outs, at = [], [], 0
    for b in prob.blocks:
        m = b.npoints
        h_in[at:at + 5 * m] = torch.from_numpy(b.state.reshape(-1))
        ins.append(api._fields_ptrs([h_in[at + v * m:at + (v + 1) * m].numpy() for v in range(5)]))
        outs.append(api._fields_ptrs([h_out[at + v * m:at + (v + 1) * m].numpy() for v in range(5)]))
        at += 5 * m
    state = {"case": dict(case), "solver": solver, "dts": _time_steps(case, prob), "ins": ins, "outs": outs,
             "h_in": h_in, "h_out": h_out}
    if prec == api.FP32_COMPENSATED:
        state["single"] = torch.empty(5 * n, dtype=torch.float32)
    return state


def _check(solver, rc):
    if rc != api.LEE_OK:
        raise api.LeeError(rc, solver.lib.last_error(solver.ctx).decode())


def run(state):
    case, solver, steps = state["case"], state["solver"], state["case"]["steps"]
    lib, ctx = solver.lib, solver.ctx
    for b, p in enumerate(state["ins"]):
        _check(solver, lib.upload_state(ctx, b, p, 0, 0.0))
    if case["kind"] == "adjoint":
        J, grad, mismatches = solver.adjoint_gradient(steps, state["dts"][0], checkpoint_every=max(8, steps // 5))
        kind = np.float32 if case["prec"] == "f32" else np.float64
        return {"J": np.asarray(J, kind), "grad": grad.astype(kind), "mismatches": int(mismatches)}
    extra = {}
    if case["kind"] == "cfl_loop":
        dt = 1e-6
        for _ in range(steps):
            dt *= 0.5 / solver.compute_cfl(dt)
            solver.advance(1, dt)
        mn, mx = solver.state_minmax()
        kind = np.float32 if case["prec"] == "f32" else np.float64
        extra = {"dt": dt, "min": mn.astype(kind), "max": mx.astype(kind)}
    elif case["kind"] == "batch":
        solver.advance_blocks(steps, state["dts"])
    else:
        solver.advance(steps, state["dts"][0])
    for b, p in enumerate(state["outs"]):
        _check(solver, lib.download_state(ctx, b, p, None, None))
    out = state["h_out"]
    if "single" in state:
        out = state["single"].copy_(out)
    return {"state": out, **extra}


def _points(case):
    """Points of each block."""
    if case["kind"] == "cylinder":
        return [case["nx"] ** 2, case["ny"] * case["nz"]]
    if case["kind"] == "batch":
        s = np.random.default_rng([case["nx"], case["ny"], case["nz"]])
        s = np.rint(np.exp(s.uniform(math.log(case["nx"]), math.log(case["ny"]), size=case["nz"])))
        return [int(n) ** 2 for n in s]
    return [case["nx"] * case["ny"] * case["nz"]]


def work(case):
    """Bytes: per RK stage the stage input read and the stage output written once, and the per-point
    coefficients (J * metrics, sponge strength, mean flow) read once; per step the filter's state
    in and out; the FP64 state in and out of the call. Operations: the stencils, the chain rule, the
    RK update and the filter's taps."""
    n = float(sum(_points(case)))
    dim = 2 if case["kind"] in ("cfl_loop", "pulse2d", "cylinder", "batch") else 3
    V, w = dim + 2, (4 if case["prec"] == "f32" else 8)
    coef = {"cfl_loop": 0, "pulse2d": 0, "batch": 0, "cylinder": 1, "curvi3d": 9, "wall3d": 15, "adjoint": 9}
    nc = coef[case["kind"]]
    wide = case.get("scheme") == "FDO11P"
    stencil = 2 * (10 if wide else 4)
    taps = 2 * (11 if wide else 9)
    step_b = n * w * (4 * (2 * V + nc) + 2 * V)
    step_f = n * (4 * (V * dim * stencil + 2 * V * dim * dim + 8 * V) + V * dim * taps)
    runs = 2 if case["kind"] == "adjoint" else 1  # a forward and a reverse sweep
    return {"bytes": runs * case["steps"] * step_b + 2 * 8 * V * n, "flops": runs * case["steps"] * step_f}


# ---- the scheme in plain FP64 torch ---------------------------------------------------------

def _fd_table(scheme):
    """Interior stencil (-h..h) and left closure rows (from the first point on) of the difference."""
    if scheme == "STANDARD_CENTRAL":
        half, rows = [8 / 12, -1 / 12], [[-1.5, 2.0, -0.5], [-0.5, 0.0, 0.5]]
    else:
        half = [0.872756993962, -0.286511173973, 0.090320001280, -0.020779405824, 0.002484594688]
        rows = [[-2.225833963270, 4.827779580575, -5.001388453836, 3.911103941646, -2.115267458633, 0.718882784412,
                 -0.115276430894],
                [-0.212932721951, -1.060320390770, 2.078926116439, -1.287179452384, 0.685176395471, -0.245320613994,
                 0.041650667189],
                [1 / 12, -8 / 12, 0.0, 8 / 12, -1 / 12],
                [-0.02625099337517627, 0.18833730683403838, -0.797921633542548, 0.0, 0.797921633542548,
                 -0.18833730683403838, 0.02625099337517627],
                [0.007650904064, -0.059463584768, 0.244678631765, -0.841570125482, 0.0, 0.841570125482,
                 -0.244678631765, 0.059463584768, -0.007650904064]]
    return [-c for c in half[::-1]] + [0.0] + half, rows, -1.0


def _filter_table(scheme):
    five = [-1 / 16, 1 / 4, 5 / 8, 1 / 4, -1 / 16]
    seven = [1 / 64, -3 / 32, 15 / 64, 11 / 16, 15 / 64, -3 / 32, 1 / 64]
    if scheme == "STANDARD_CENTRAL":
        d, rows = [35 / 128, -7 / 32, 7 / 64, -1 / 32, 1 / 256], [[1.0], [0.0, 1.0], five, seven]
    else:
        d = [0.215044884112, -0.187772883589, 0.123755948787, -0.059227575576, 0.018721609157, -0.002999540835]
        nine = [0.008228661760, -0.045211119360, 0.120007591680, -0.204788880640, 0.243527493120, -0.204788880640,
                0.120007591680, -0.045211119360, 0.008228661760]
        rows = [[1.0], [0.0, 1.0], five, seven, [(1.0 if s == 4 else 0.0) - c for s, c in enumerate(nine)]]
    half = [-c for c in d[1:]]
    return half[::-1] + [1.0 - d[0]] + half, rows, 1.0


def _line_matrix(table, n, blank=None):
    """The operator on one grid line of n points as a dense matrix. blank: 1 hole, -1 receiver;
    closure rows stand on both sides of a hole (after a receiver; after a plain fluid point there is
    none), and a hole after a hole gives zero."""
    stencil, rows, mirror = table
    h = len(stencil) // 2
    m = np.zeros((n, n))
    for i in range(h, n - h):
        m[i, i - h:i + h + 1] = stencil
    for r, row in enumerate(rows):
        m[r, :] = 0.0
        m[r, :len(row)] = row
    for r, row in enumerate(rows):
        m[n - 1 - r, :] = 0.0
        m[n - 1 - r, n - len(row):] = mirror * np.asarray(row)[::-1]
    if blank is None:
        return m
    last = blank[0]
    for i in range(n):
        if blank[i] == 1:
            if last == 1:
                m[i] = 0.0
            elif last == -1 and i > 0:
                for r, row in enumerate(rows):
                    m[i - 1 - r] = 0.0
                    m[i - 1 - r, i - len(row):i] = mirror * np.asarray(row)[::-1]
        elif last == 1:
            for r, row in enumerate(rows):
                m[i + r] = 0.0
                m[i + r, i:i + len(row)] = row
        last = blank[i]
    return m


class _Operator:
    """A table applied along the directions of a block, to fields of shape (..., nz, ny, nx)."""

    def __init__(self, table, dims, blank=None):
        self.dims = dims
        self.mat = [torch.tensor(_line_matrix(table, n), device=DEVICE) if n > 1 else None for n in dims]
        self.own = ([], [])  # (line, matrix) of lines with holes, 2-D blocks only
        if blank is not None:
            b = blank[0]
            for j in np.nonzero((b == 1).any(axis=1))[0]:
                self.own[0].append((int(j), torch.tensor(_line_matrix(table, dims[0], b[j]), device=DEVICE)))
            for i in np.nonzero((b == 1).any(axis=0))[0]:
                self.own[1].append((int(i), torch.tensor(_line_matrix(table, dims[1], b[:, i]), device=DEVICE)))

    def __call__(self, f, d):
        if self.mat[d] is None:
            return None
        if d == 0:
            out = f @ self.mat[0].T
            for j, m in self.own[0]:
                out[..., j, :] = f[..., j, :] @ m.T
            return out
        if d == 1:
            out = self.mat[1] @ f
            for i, m in self.own[1]:
                out[..., :, i] = f[..., :, i] @ m.T
            return out
        s = f.shape
        return (self.mat[2] @ f.reshape(*s[:-2], s[-2] * s[-1])).reshape(s)


class _Block:
    def __init__(self, prob, b):
        blk = prob.blocks[b]
        to = lambda a: torch.tensor(a, dtype=torch.float64, device=DEVICE)  # noqa: E731
        self.dim, self.dims = prob.num_dim, blk.dims
        self.xyz = [to(a) for a in (blk.x, blk.y, blk.z)]
        self.mean = to(blk.mean)
        blank = None
        if prob.overset is not None:
            blank = np.zeros(blk.x.shape, int)
            o = prob.overset
            for who, at, what in ((o.hole_block, o.hole_ijk, 1), (o.recv_block, o.recv_ijk, -1)):
                at = np.asarray(at)[np.asarray(who) == b]
                blank[at[:, 2], at[:, 1], at[:, 0]] = what
            blank = blank if (blank != 0).any() else None
        holes = blank if blank is not None and (blank == 1).any() else None
        self.fluid = None if holes is None else to((holes != 1).astype(float))
        self.counted = None if blank is None else torch.tensor(blank == 0, device=DEVICE)
        fd, flt = _fd_table(prob.fd_scheme), _filter_table(prob.filter_scheme)
        self.d = _Operator(fd, blk.dims, holes)
        self.f = _Operator(flt, blk.dims, holes)
        self._metrics(_Operator(fd, blk.dims) if holes is not None else self.d)
        self.edge = torch.tensor(fd[1][0], dtype=torch.float64, device=DEVICE)
        D = range(self.dim)
        self.varies = [bool((m.max() - m.min()) > 0) for m in self.mean]
        self.grad = [[self.cart(self.mean[v], j) if self.varies[v] else None for j in D] for v in range(5)]
        self.rhobar = (GAMMA * self.mean[4]) ** (1.0 / GAMMA) * torch.exp(-self.mean[0])
        self.shear = any(self.varies[1 + i] for i in D)
        self.sigma = torch.zeros_like(self.xyz[0])
        self.lines = []
        for bd in prob.boundaries:
            if bd.block != b:
                continue
            if bd.kind != "sponge_freund_ambient":
                self.lines.append(bd)
                continue
            box = tuple(slice(bd.lo[q], bd.hi[q] + 1) for q in (2, 1, 0))
            sg = bd.sigma if bd.sigma is not None else builders.sponge_sigma(prob, bd)
            self.sigma[box] += to(np.asarray(sg).reshape(self.sigma[box].shape))
        self.source, self.amp = None, lambda t: 0.0
        mono = blk.monopole or prob.source_monopole()
        if mono is not None:
            x0, y0, z0, a, om, hw, ramp = mono
            r2 = (self.xyz[0] - x0) ** 2 + (self.xyz[1] - y0) ** 2 + (self.xyz[2] - z0) ** 2
            self.source = torch.exp(-math.log(2.0) / hw ** 2 * r2)
            self.amp = lambda t: (a * (GAMMA - 1.0) * math.sin(om * t) *
                                  (math.sin(0.5 * math.pi * t / ramp) ** 2 if 0.0 < ramp and t < ramp else 1.0))
        if prob.distributed is not None:
            om = prob.distributed.omega
            self.amp = lambda t: (GAMMA - 1.0) * math.sin(om * t)

    def _metrics(self, op):
        """Thomas-Lombard products: met[l][i] = (1/J) d xi_l / d x_i."""
        x = self.xyz
        if self.dim == 2:
            d = [[op(x[i], l) for l in range(2)] for i in range(2)]
            self.met = [[d[1][1], -d[0][1]], [-d[1][0], d[0][0]]]
            inv = d[0][0] * d[1][1] - d[0][1] * d[1][0]
        else:
            d = [[op(x[i], l) for l in range(3)] for i in range(3)]
            # (1/J) d xi_l / d x_i = d_m (d_k a  b)... cyclic in both the directions and the coordinates
            self.met = [[None] * 3 for _ in range(3)]
            for l in range(3):
                m, n = (l + 1) % 3, (l + 2) % 3
                for i in range(3):
                    p, q = (i + 1) % 3, (i + 2) % 3
                    if i == 2:  # coordinate pair (x, y): products with y
                        p, q = 0, 1
                        s = 1.0
                    elif i == 1:  # (z, x) written as (x, z) with the sign turned
                        p, q = 0, 2
                        s = -1.0
                    else:
                        s = 1.0
                    self.met[l][i] = s * (op(d[p][m] * x[q], n) - op(d[p][n] * x[q], m))
            inv = (d[0][0] * (d[1][1] * d[2][2] - d[1][2] * d[2][1])
                   - d[0][1] * (d[1][0] * d[2][2] - d[1][2] * d[2][0])
                   + d[0][2] * (d[1][0] * d[2][1] - d[1][1] * d[2][0]))
        self.jac = 1.0 / inv

    def cart(self, f, j):
        return self.jac * sum(self.met[l][j] * self.d(f, l) for l in range(self.dim))

    def rho(self, q):
        """rho' / rho_bar."""
        return q[4] / (GAMMA * self.mean[4]) - q[0]

    def rhs(self, q, t, rho):
        D, m = range(self.dim), self.mean
        g = [self.d(q, l) for l in D]
        dx = lambda v, j: self.jac * sum(self.met[l][j] * g[l][v] for l in D)  # noqa: E731
        out = []
        conv = [1 + j for j in D if self.varies[1 + j] or bool(m[1 + j].abs().max() > 0)]
        div = sum(dx(1 + j, j) for j in D)
        for v in range(5):
            if v == 3 and self.dim == 2:
                out.append(torch.zeros_like(q[3]))
                continue
            r = -self.sigma * q[v]
            for u in conv:
                r = r - m[u] * dx(v, u - 1)
            if self.varies[v]:
                for j in D:
                    w = q[1 + j] + rho * m[1 + j] if 1 <= v <= 3 else q[1 + j]
                    r = r - w * self.grad[v][j]
            if 1 <= v <= 3:
                r = r - dx(4, v - 1) / self.rhobar
            if v == 4:
                r = r - GAMMA * m[4] * div
                for j in D:
                    if self.varies[1 + j]:
                        r = r - GAMMA * q[4] * self.grad[1 + j][j]
                if self.source is not None:
                    r = r + self.amp(t) * self.source
            out.append(r)
        return torch.stack(out)

    def boundaries(self, q):
        for bd in self.lines:
            ax = 3 - bd.dir
            n = q.shape[ax]
            at = lambda s: q.select(ax, s if bd.end == 0 else n - 1 - s)  # noqa: E731,B023
            face = at(0)
            neu = range(5) if bd.kind == "neumann" else (0, 4)
            new = {v: -sum(self.edge[s] * at(s)[v] for s in range(1, len(self.edge))) / self.edge[0] for v in neu}
            if bd.kind == "wall_slip_kinematic":
                cut = lambda f: f.select(ax - 1, 0 if bd.end == 0 else n - 1)  # noqa: E731,B023
                D = range(self.dim)
                M = [[cut(self.met[l][i]) for i in D] for l in D]
                con = [sum(M[l][i] * face[1 + i] for i in D) if l != bd.dir else 0.0 for l in D]
                if self.dim == 2:
                    adj = [[M[1][1], -M[0][1]], [-M[1][0], M[0][0]]]
                else:
                    adj = [[M[(l + 1) % 3][(i + 1) % 3] * M[(l + 2) % 3][(i + 2) % 3]
                            - M[(l + 1) % 3][(i + 2) % 3] * M[(l + 2) % 3][(i + 1) % 3] for l in D] for i in D]
                for i in D:
                    new[1 + i] = cut(self.jac) * sum(adj[i][l] * con[l] for l in D)
            for v, val in new.items():
                face[v] = val

    def filtered(self, q):
        for d in range(self.dim):
            q = self.f(q, d)
        return q if self.fluid is None else q * self.fluid

    def cfl(self, dt):
        D, m = range(self.dim), self.mean
        con = [sum(self.met[l][i] * m[1 + i] for i in D) for l in D]
        c = sum(torch.trunc(con[l] * self.met[l][i]).abs() for l in D for i in D)
        sound = torch.sqrt(GAMMA * m[4] / self.rhobar)
        c = (c + sound * torch.sqrt(sum(self.met[l][i] ** 2 for l in D for i in D))) * dt * self.jac
        return float((c if self.counted is None else c[self.counted]).max())


class _Overset:
    def __init__(self, o, blocks):
        self.parts = []
        wt = np.asarray(o.weights, float).reshape(len(o.recv_block), -1)
        wt = wt / wt.sum(axis=1, keepdims=True)
        rb, db = np.asarray(o.recv_block), np.asarray(o.donor_block)
        dev = lambda a: torch.tensor(a, device=DEVICE)  # noqa: E731
        for r in range(len(blocks)):
            for d in range(len(blocks)):
                sel = (rb == r) & (db == d)
                if not sel.any():
                    continue
                ri, di = np.asarray(o.recv_ijk)[sel], np.asarray(o.donor_ijk)[sel]
                rx, ry, _ = blocks[r].dims
                nx, ny, _ = blocks[d].dims
                off = [a + nx * (b + ny * c) for c in range(o.width[2]) for b in range(o.width[1])
                       for a in range(o.width[0])]
                dl = di[:, 0] + nx * (di[:, 1] + ny * di[:, 2])
                self.parts.append((r, d, dev(ri[:, 0] + rx * (ri[:, 1] + ry * ri[:, 2])),
                                   dev(dl[:, None] + np.asarray(off)[None, :]), dev(wt[sel])))

    def __call__(self, qs):
        new = [(r, rl, (qs[d].reshape(5, -1)[:, dl] * w).sum(-1)) for r, d, rl, dl, w in self.parts]
        for r, rl, v in new:
            qs[r].reshape(5, -1)[:, rl] = v


_RK4 = ((1 / 6, 0.0, 0.5), (1 / 3, 0.5, 0.5), (1 / 3, 0.5, 1.0), (1 / 6, 1.0, 0.0))  # b, c, a


def _step(blocks, overset, qs, rhos, t, dt):
    """One RK4 step of all blocks ending at time t (the scheme's clock runs ahead: stage times are t + c dt)."""
    total, z = [q for q in qs], [q for q in qs]
    for s, (b, c, a) in enumerate(_RK4):
        for k, blk in enumerate(blocks):
            rho = (rhos[k] if s == 0 and rhos[k] is not None else blk.rho(z[k])) if blk.shear else None
            r = dt * blk.rhs(z[k], t + c * dt, rho)
            total[k] = total[k] + b * r
            z[k] = qs[k] + a * r
            if blk.fluid is not None:
                total[k], z[k] = total[k] * blk.fluid, z[k] * blk.fluid
        target = total if s == 3 else z
        for blk, q in zip(blocks, target):
            blk.boundaries(q)
        if overset is not None:
            overset(target)
    rhos = [blk.rho(q) if blk.shear else None for blk, q in zip(blocks, total)]
    return [blk.filtered(q) for blk, q in zip(blocks, total)], rhos


def _lattice(src, dims):
    """The source's box of grid points and the matrices that prolong the lattice onto it."""
    mats, box = [], []
    for d in range(3):
        o, h, c = src.origin[d], src.spacing[d], src.amplitudes.shape[2 - d]
        lo, hi = max(0, math.ceil(o)), min(dims[d] - 1, math.floor(o + (c - 1) * h))
        m = np.zeros((hi - lo + 1, c))
        for r, i in enumerate(range(lo, hi + 1)):
            u = (i - o) / h
            p = min(max(int(math.floor(u)), 0), c - 2)
            m[r, p], m[r, p + 1] = 1.0 - (u - p), u - p
        mats.append(torch.tensor(m, device=DEVICE))
        box.append(slice(lo, hi + 1))
    return mats, box


def exact(case, seed):
    torch.backends.cuda.matmul.allow_tf32 = False
    prob = _problem(case, seed)
    steps, dts = case["steps"], _time_steps(case, prob)
    start = [torch.tensor(b.state, device=DEVICE) for b in prob.blocks]
    if case["kind"] == "adjoint":
        return _exact_gradient(prob, start[0], steps, dts[0])
    flat = []
    extra = {}
    if case["kind"] == "batch":
        for b, q in enumerate(start):
            blk = _Block(prob, b)
            flat.append(_march([blk], None, [q], steps, [dts[b]] * steps)[0])
    else:
        blocks = [_Block(prob, b) for b in range(len(start))]
        overset = _Overset(prob.overset, blocks) if prob.overset is not None else None
        times = [dts[0]] * steps
        if case["kind"] == "cfl_loop":
            times, dt = [], 1e-6
            for _ in range(steps):
                dt *= 0.5 / blocks[0].cfl(dt)
                times.append(dt)
        flat = _march(blocks, overset, start, steps, times)
        if case["kind"] == "cfl_loop":
            q = flat[0].reshape(5, -1)
            extra = {"dt": times[-1], "min": q.min(1).values.cpu().numpy(), "max": q.max(1).values.cpu().numpy()}
    return {"state": torch.cat([q.reshape(-1) for q in flat]).cpu(), **extra}


def _march(blocks, overset, qs, steps, dts):
    rhos, t = [None] * len(qs), 0.0
    with torch.no_grad():
        for n in range(steps):
            t += dts[n]
            qs, rhos = _step(blocks, overset, qs, rhos, t, dts[n])
    return qs


def _exact_gradient(prob, q, steps, dt):
    """The objective and its gradient by reverse mode over the forward scheme, one step at a time."""
    blk = _Block(prob, 0)
    src = prob.distributed
    mats, box = _lattice(src, blk.dims)
    mic = torch.tensor(prob.microphones.l0, device=DEVICE)
    wt = prob.microphones.weight
    amps = torch.tensor(src.amplitudes, device=DEVICE, requires_grad=True)
    field = torch.einsum("za,yb,xc,abc->zyx", mats[2], mats[1], mats[0], amps)
    spread = torch.zeros_like(blk.sigma)
    spread[box[2], box[1], box[0]] = field.detach()
    blk.source = spread
    J, t, p = 0.0, 0.0, []
    with torch.no_grad():
        for n in range(steps):
            t += dt
            q = _step([blk], None, [q], [None], t, dt)[0][0]
            p.append(q[4].reshape(-1)[mic].clone())
            J += wt * float((p[-1] ** 2).sum())
    # the step is affine in (state, source field): its transpose needs no forward state
    lam, gfield = torch.zeros_like(q), torch.zeros_like(spread)
    for n in reversed(range(steps)):
        lam[4].reshape(-1)[mic] += 2.0 * wt * p[n]
        tn = dt * 0.0
        for _ in range(n + 1):
            tn += dt
        z = torch.zeros_like(q, requires_grad=True)
        blk.source = spread.clone().requires_grad_(True)
        out = _step([blk], None, [z], [None], tn, dt)[0][0]
        gz, gs = torch.autograd.grad(out, (z, blk.source), lam)
        lam, gfield = gz, gfield + gs
    grad, = torch.autograd.grad(field, amps, gfield[box[2], box[1], box[0]])
    return {"J": J, "grad": grad.detach().cpu(), "mismatches": None}
