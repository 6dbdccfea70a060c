"""The work that users of this framework have it do, as cases to measure.

Four kinds of call, each through the Python binding's public entry points:

  solver  one LBM-IB problem (lbib.Solver): a number of time steps, then the
          fields and the sheets read back, as a program does that writes
          its dumps every so many steps;
  sweep   many uneven problems as one batch (lbib.Batch): a number of steps,
          then the stop codes and every sheet, which is what the parameter
          sweeps record;
  train   the sweep surrogate's training (lbib.MLP): a run of Adam steps over
          an epoch's minibatches, then the parameters;
  screen  its use: every member of an ensemble evaluated on all the points.

Lengths are in lattice units and axes the library's own (x is the flow
direction).  Inputs follow from the seed alone: the physics a little off the
case's nominal values, sheets smoothly deformed with some node noise, random
network weights and data.  Inflow speeds and sheet stiffnesses are those
with which the explicit fluid-sheet coupling stays stable for tens of
thousands of steps, so that a state can be advanced again and again.
"""
import math
import os
import sys
from dataclasses import dataclass
from typing import List

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "distributed-lb-ib_b200"))
import lbib  # noqa: E402

POP_BYTES = {"f64": 8, "f32": 4, "f32-flow": 4, "f16": 2, "f16-flow": 2, "bf16": 2, "bf16-flow": 2}
PERIODIC_Z, REST_START, PIN_ROW0 = 0x100, 0x200, 0x400   # LBIB_OPT_* of include/lbib.h


# ---- the cases --------------------------------------------------------------

def _solver(name, nx, ny, nz, rows, cols, steps, precision="f64", sheets=1, u=0.0005, tau=0.6, ks=1e-4, kb=1e-5,
            cube=4, options=0, autotune=False):
    return {"name": name, "kind": "solver", "nx": nx, "ny": ny, "nz": nz, "cube": cube, "rows": rows, "cols": cols,
            "sheets": sheets, "steps": steps, "precision": precision, "u": u, "tau": tau, "ks": ks, "kb": kb,
            "options": options, "autotune": autotune}


def _sweep(name, n, sizes, steps, precision):
    return {"name": name, "kind": "sweep", "problems": n, "sizes": sizes, "steps": steps, "precision": precision}


def _train(name, widths, batch, steps):
    return {"name": name, "kind": "train", "widths": widths, "batch": batch, "steps": steps}


def _screen(name, widths, batch, points, members):
    return {"name": name, "kind": "screen", "widths": widths, "batch": batch, "points": points, "members": members}


def listed():
    return [
        # the smallest useful channel, read back every few steps: latency and launches
        _solver("channel_64_f64", 64, 32, 32, 16, 16, 8, u=0.0002, ks=5e-5, kb=5e-6),
        # the solver's own reference size (128 x 64 x 64, a 52 x 52 sheet); fits L2
        _solver("channel_128_f64", 128, 64, 64, 52, 52, 50),
        # the same run in the 16-bit storage form, without a trial of the kernel variants
        _solver("channel_128_f16", 128, 64, 64, 52, 52, 50, "f16-flow"),
        # odd extents, two pinned flaps of uneven rows and columns, periodic z, a start from rest
        _solver("flaps_100_f64", 100, 55, 75, 37, 29, 24, sheets=2, cube=5,
                options=PERIODIC_Z | REST_START | PIN_ROW0),
        # a mid-size run with two sheets in 32-bit storage
        _solver("sheets_256_f32", 256, 128, 128, 104, 104, 20, "f32", sheets=2, u=0.002, ks=2e-4, kb=2e-5),
        # the benchmark size, 512 x 256 x 256 with a 208 x 208 sheet: the drop-in precision ...
        _solver("channel_512_f64", 512, 256, 256, 208, 208, 50, u=0.01, ks=2e-3, kb=2e-4),
        # ... and the 16-bit form as a long run sets it up, its kernel variant tried out first
        _solver("channel_512_f16", 512, 256, 256, 208, 208, 50, "f16-flow", u=0.01, ks=2e-3, kb=2e-4, autotune=True),
        # the few re-runs that a screened sweep sends back, in the judge's precision
        _sweep("rerun_24_f64", 24, 3, 20, "f64"),
        # a plain parameter sweep in the 16-bit form
        _sweep("sweep_128_f16", 128, 1, 50, "f16-flow"),
        # training the displacement surrogate: the tool's own widths and minibatch
        _train("train_256x4", "5,256,256,256,256,192", 1024, 16),
        # the stop classifier's small net on a ragged minibatch
        _train("train_64x2", "4,64,64,1", 1000, 16),
        # screening 2048 held-out points with five members
        _screen("screen_2048", "5,256,256,256,256,192", 1024, 2048, 5),
    ]


def _log_int(rng, lo, hi, step=1):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))


def draw(rng):
    kind = rng.choice(["solver"] * 11 + ["sweep"] * 4 + ["train"] * 3 + ["screen"] * 2)
    if kind == "solver":
        cube = rng.choice([4, 4, 4, 4, 5, 6])
        lo = -(-24 // cube) * cube
        whole = {4: 4, 5: 20, 6: 12}[cube]          # x takes whole cubes and whole tiles of 4
        nx = max(60, _log_int(rng, 48, 512) // whole * whole)
        # nx >= nz: the reference's loop-bound slips stay idle
        ny, nz = (max(lo, _log_int(rng, 24, min(nx, 256)) // cube * cube) for _ in range(2))
        sites = nx * ny * nz
        steps = min(_log_int(rng, 4, 64), max(2, 600_000_000 // sites))
        c = _solver("", nx, ny, nz, rng.randint(8, max(9, int(1.5 * ny))), rng.randint(8, max(9, int(1.5 * nz))), steps,
                    rng.choice(["f64"] * 5 + ["f16-flow"] * 4 + ["f32", "f32-flow", "f16", "bf16-flow"]),
                    rng.choice([1, 1, 1, 2]), rng.choice([0.0002, 0.0005, 0.001]), rng.choice([0.6, 0.7, 0.8]),
                    1e-4, 1e-5, cube, rng.choice([0, 0, 0, PERIODIC_Z, REST_START, PIN_ROW0, PERIODIC_Z | PIN_ROW0]))
        if nx < 96:
            c["u"] = 0.0002
    elif kind == "sweep":
        n = _log_int(rng, 4, 128)
        c = _sweep("", n, rng.randint(1, 10 ** 6), _log_int(rng, 6, 60), rng.choice(["f64", "f16-flow", "f16-flow", "f32"]))
    elif kind == "train":
        h = _log_int(rng, 32, 320)
        w = [rng.randint(3, 8)] + [h] * rng.randint(1, 5) + [rng.choice([1, 3, 48, 192, 200])]
        c = _train("", ",".join(map(str, w)), _log_int(rng, 64, 2048), rng.randint(4, 16))
    else:
        h = _log_int(rng, 32, 320)
        w = [rng.randint(3, 8)] + [h] * rng.randint(1, 5) + [rng.choice([1, 3, 48, 192, 200])]
        c = _screen("", ",".join(map(str, w)), _log_int(rng, 128, 1024), _log_int(rng, 100, 4096), rng.randint(1, 5))
    del c["name"]
    return c


# ---- inputs -----------------------------------------------------------------

@dataclass
class SheetSpec:
    rows: int
    cols: int
    width: float
    height: float
    x0: float
    y0: float
    z0: float


@dataclass
class ChannelSpec:
    nx: int
    ny: int
    nz: int
    cube_size: int
    sheets: List[SheetSpec]
    tau: float
    u_l: float
    Ks_l: float
    Kb_l: float
    compat: int


def _channel(case, seed):
    """The problem, and every sheet's deformed positions [rows, cols, 3]."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    rows, cols = case["rows"], case["cols"]
    # node spacing 0.5, closer where the sheet would not clear the walls
    h = min(0.5 * (rows - 1), ny - 14.0)
    w = min(0.5 * (cols - 1), nz - 14.0)
    specs, pos = [], []
    for k in range(case["sheets"]):
        x0 = float(int(nx * (0.16 + 0.22 * k)))
        s = SheetSpec(rows, cols, w, h, x0, (ny - 1) / 2.0 - h / 2.0, (nz - 1) / 2.0 - w / 2.0)
        specs.append(s)
        r, c = np.meshgrid(np.linspace(0.0, 1.0, rows), np.linspace(0.0, 1.0, cols), indexing="ij")
        p = np.stack([np.full_like(r, s.x0), s.y0 + h * r, s.z0 + w * c], axis=-1)
        for d in range(3):
            for _ in range(3):
                a, b, phase = rng.integers(0, 3), rng.integers(0, 3), rng.uniform(0, 2 * math.pi)
                p[..., d] += rng.uniform(-0.25, 0.25) * np.cos(math.pi * (a * r + b * c) + phase)
        p += rng.uniform(-0.01, 0.01, p.shape)
        pos.append(p)
    scale = rng.uniform(0.9, 1.1, 3)
    tau = case["tau"] + rng.uniform(0.0, 0.05)
    spec = ChannelSpec(nx, ny, nz, case["cube"], specs, float(tau), float(case["u"] * scale[0]),
                       float(case["ks"] * scale[1]), float(case["kb"] * scale[2]), lbib.COMPAT_ALL | case["options"])
    return spec, pos


def _problems(case, seed):
    """Sizes from the case, physics from the seed, in the ranges of the sweep
    tool's calmer runs (those that reach their end)."""
    sizes, rng = np.random.default_rng(case["sizes"]), np.random.default_rng(seed)
    out = []
    for _ in range(case["problems"]):
        nx = int(sizes.choice((48, 64, 96, 128, 192)))
        ny, nz = (int(v) for v in sizes.choice((32, 48, 64), 2))
        side = int(sizes.integers(8, 41))
        ks, kb = 10 ** rng.uniform(-4.3, -3.7), 10 ** rng.uniform(-5.3, -4.7)
        w = 0.5 * (side - 1)
        out.append(lbib.Problem(nx, ny, nz, float(rng.uniform(0.6, 0.9)), float(rng.uniform(0.0003, 0.0008)),
                                float(ks), float(kb), side, side, w, w, nx / 6.0, (ny - 1) / 2.0 - w / 2.0,
                                (nz - 1) / 2.0 - w / 2.0, 1))
    return out


def _widths(case):
    return [int(w) for w in case["widths"].split(",")]


def _weights(widths, rng):
    """One network's parameters in the library's order: W [out][in], b [out] per layer."""
    parts = []
    for a, b in zip(widths[:-1], widths[1:]):
        parts.append(rng.uniform(-1, 1, a * b) * math.sqrt(6.0 / a))
        parts.append(rng.uniform(-0.1, 0.1, b))
    return np.concatenate(parts).astype(np.float32)


def _train_data(case, seed):
    """Weights, and an epoch of four minibatches: smooth targets of the inputs."""
    rng = np.random.default_rng(seed)
    w = _widths(case)
    p = _weights(w, rng)
    X = rng.uniform(-1, 1, (4 * case["batch"], w[0])).astype(np.float32)
    A, B = rng.normal(0, 1, (w[0], 24)), rng.normal(0, 0.4, (24, w[-1]))
    T = (np.sin(X @ A) @ B).astype(np.float32)
    return p, X, T


LEARNING_RATE = 1e-3


# ---- what a user's program has in hand, and one pass ------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "solver":
        spec, pos = _channel(case, seed)
        s = lbib.Solver(spec, case["precision"])
        if case["autotune"]:
            s.autotune(4)
        for k, p in enumerate(pos):
            rec = s.sheet(k)
            rec[..., :3] = p
            s.set_sheet(k, rec)
        # page-locked, as a program keeps them that reads the fields more than once
        out = [torch.empty(s.N, dtype=torch.float64, pin_memory=True).numpy() for _ in range(4)]
        return {"kind": kind, "solver": s, "steps": case["steps"], "out": out}
    if kind == "sweep":
        b = lbib.Batch(_problems(case, seed), case["precision"], compat=0)
        return {"kind": kind, "batch": b, "steps": case["steps"]}
    if kind == "train":
        p, X, T = _train_data(case, seed)
        net = lbib.MLP(_widths(case), max_batch=case["batch"], seed=seed % 1000)
        net.set_params(p)
        cut = lambda a: [c.contiguous() for c in torch.from_numpy(a).cuda().split(case["batch"])]  # noqa: E731
        return {"kind": kind, "net": net, "X": cut(X), "T": cut(T), "steps": case["steps"]}
    rng = np.random.default_rng(seed)
    w = _widths(case)
    nets = []
    for m in range(case["members"]):
        net = lbib.MLP(w, max_batch=case["batch"], seed=m)
        net.set_params(_weights(w, rng))
        nets.append(net)
    X = torch.from_numpy(rng.uniform(-1, 1, (case["points"], w[0])).astype(np.float32)).cuda()
    return {"kind": kind, "nets": nets, "X": X}


def run(state):
    kind = state["kind"]
    if kind == "solver":
        s = state["solver"]
        s.run(state["steps"])
        rho, ux, uy, uz = s.moments(state["out"])
        return {"rho": rho, "ux": ux, "uy": uy, "uz": uz, "sheets": [s.sheet(k) for k in range(len(s.case.sheets))]}
    if kind == "sweep":
        b = state["batch"]
        b.run(state["steps"])
        codes, _ = b.status()
        return {"codes": codes, "sheets": np.concatenate([b.sheet(k).ravel() for k in range(len(b))])}
    if kind == "train":
        net, X, T = state["net"], state["X"], state["T"]
        for i in range(state["steps"]):
            net.train_step(X[i % len(X)], T[i % len(T)], LEARNING_RATE)
        return net.params()
    X = state["X"]
    return [torch.cat([net.forward(X[c:c + net.max_batch].contiguous()) for c in range(0, X.shape[0], net.max_batch)])
            for net in state["nets"]]


# ---- the least work ---------------------------------------------------------

STEP_FLOPS = 250   # moments, equilibria and relaxation of one D3Q19 cell
NODE_FLOPS = 900   # forces, 12 delta factors, 64 cells of spread and of interpolation


def work(case):
    kind = case["kind"]
    if kind == "solver":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        cells = (nx - 4) * (ny - 4) * (nz - 4)
        nodes = case["sheets"] * case["rows"] * case["cols"]
        per_step = 38 * POP_BYTES[case["precision"]] * cells + 24 * 8 * nodes
        return {"bytes": case["steps"] * per_step + 32 * nx * ny * nz + 96 * nodes,
                "flops": case["steps"] * (STEP_FLOPS * cells + NODE_FLOPS * nodes)}
    if kind == "sweep":
        ps = _problems(case, 0)
        cells = sum((p.nx - 4) * (p.ny - 4) * (p.nz - 4) for p in ps)
        nodes = sum(p.rows * p.cols for p in ps)
        per_step = 38 * POP_BYTES[case["precision"]] * cells + 24 * 8 * nodes
        return {"bytes": case["steps"] * per_step + 96 * nodes,
                "flops": case["steps"] * (STEP_FLOPS * cells + NODE_FLOPS * nodes)}
    w = _widths(case)
    params = sum(a * b + b for a, b in zip(w[:-1], w[1:]))
    mul = sum(a * b for a, b in zip(w[:-1], w[1:]))
    if kind == "train":
        # master weights and both Adam moments read and written, inputs and targets read
        return {"bytes": case["steps"] * (24 * params + 4 * case["batch"] * (w[0] + w[-1])) + 4 * params,
                "flops": case["steps"] * 6 * mul * case["batch"]}
    return {"bytes": case["members"] * (2 * params + 4 * case["points"] * (w[0] + w[-1])),
            "flops": case["members"] * 2 * mul * case["points"]}


# ---- the same results in 64 bits, by plain torch ----------------------------

# the D3Q19 velocities in the library's order (x, y, z)
C = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 0, 1), (0, 0, -1), (0, -1, 0), (0, 1, 0), (1, 0, 1), (-1, 0, -1), (1, 0, -1),
     (-1, 0, 1), (0, -1, 1), (0, 1, -1), (0, 1, 1), (0, -1, -1), (1, -1, 0), (-1, 1, 0), (1, 1, 0), (-1, -1, 0)]
OPP = [0] + [q + 1 if q % 2 else q - 1 for q in range(1, 19)]
WEIGHT = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12


def _equilibrium(q, rho, ux, uy, uz, usq):
    cu = C[q][0] * ux + C[q][1] * uy + C[q][2] * uz
    return WEIGHT[q] * rho * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * usq)


def _bend(p, coef, dim, slip):
    """Bending force along one direction of a sheet [rows, cols, 3].  `slip`:
    along a fiber the x component at the last node but one takes its own
    position for the one two nodes back."""
    p = p.transpose(0, dim)
    n = p.shape[0]
    b = torch.empty_like(p)
    b[0] = -p[2] + 2 * p[1] - p[0]
    b[1] = -p[3] + 4 * p[2] - 5 * p[1] + 2 * p[0]
    b[2:n - 2] = -p[4:] + 4 * p[3:n - 1] - 6 * p[2:n - 2] + 4 * p[1:n - 3] - p[:n - 4]
    last = p[n - 4].clone()
    if slip:
        last[..., 0] = p[n - 2][..., 0]
    b[n - 2] = 2 * p[n - 1] - 5 * p[n - 2] + 4 * p[n - 3] - last
    b[n - 1] = -p[n - 1] + 2 * p[n - 2] - p[n - 3]
    return coef * b.transpose(0, dim)


def _stretch(p, coef, rest, dim):
    """Stretching force along one direction; the last node's tangent points
    from its neighbour, as the step has it."""
    p = p.transpose(0, dim)
    t = p[1:] - p[:-1]
    length = t.norm(dim=-1, keepdim=True)
    f = (length - rest) * t / length
    s = torch.empty_like(p)
    s[0], s[-1] = f[0], f[-1]
    s[1:-1] = f[1:] - f[:-1]
    return coef * s.transpose(0, dim)


class _Flow:
    """The time step of one problem in 64-bit torch."""

    def __init__(self, spec, pos, device):
        self.c, self.dev = spec, device
        f64 = {"dtype": torch.float64, "device": device}
        n = (spec.nz, spec.ny, spec.nx)
        self.rho = torch.ones(n, **f64)
        self.u = [torch.full(n, spec.u_l, **f64), torch.zeros(n, **f64), torch.zeros(n, **f64)]
        if spec.compat & REST_START:
            self.u[0][:, :, 3:spec.nx - 3] = 0.0
        cells = tuple(slice(2, k - 2) for k in n)
        self.cells = cells
        ux = self.u[0][cells]
        self.f = torch.stack([_equilibrium(q, 1.0, ux, 0.0, 0.0, ux * ux) for q in range(19)])
        self.plane = [float(_equilibrium(q, 1.0, spec.u_l, 0.0, 0.0, spec.u_l ** 2)) for q in range(19)]
        self.pos = [torch.from_numpy(np.ascontiguousarray(p)).to(**f64) for p in pos]
        self.force = [None] * len(pos)

    def _stencil(self, p):
        """Cell indices [S, 64] and delta factors of nodes [S, 3], 1/64 included."""
        c = self.c
        start = (p - 2).floor() + 1
        o = torch.arange(4, dtype=torch.float64, device=self.dev)
        g = start[:, :, None] + o
        w = 1 + torch.cos(math.pi / 2 * (g - p[:, :, None]))
        g = g.long()
        idx = (g[:, 2, None, None, :] * c.ny + g[:, 1, None, :, None]) * c.nx + g[:, 0, :, None, None]
        wt = w[:, 0, :, None, None] * w[:, 1, None, :, None] * w[:, 2, None, None, :] / 64
        return idx.reshape(len(p), 64), wt.reshape(len(p), 64)

    def step(self):
        c = self.c
        spread = [torch.zeros(c.nz * c.ny * c.nx, dtype=torch.float64, device=self.dev) for _ in range(3)]
        for k, (s, p) in enumerate(zip(c.sheets, self.pos)):
            ds1, ds2 = s.width / (s.cols - 1), s.height / (s.rows - 1)
            kb = c.Kb_l / ds2 ** 3
            bend = _bend(p, kb, 1, bool(c.compat & lbib.COMPAT_BEND_X_BUG)) + _bend(p, kb, 0, False)
            stretch = _stretch(p, c.Ks_l / ds1 ** 2, ds1, 1) + _stretch(p, c.Ks_l / ds2 ** 2, ds2, 0)
            self.force[k] = (bend, stretch, bend + stretch)
            idx, w = self._stencil(p.reshape(-1, 3))
            e = self.force[k][2].reshape(-1, 3)
            for d in range(3):
                spread[d].index_add_(0, idx.reshape(-1), (w * e[:, d, None]).reshape(-1))
        F = [v.view(c.nz, c.ny, c.nx)[self.cells] for v in spread]
        rho = self.rho[self.cells]
        u = [v[self.cells] for v in self.u]
        usq = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
        uF = u[0] * F[0] + u[1] * F[1] + u[2] * F[2]
        guo = 1 - 1 / (2 * c.tau)
        for q in range(19):
            cu = C[q][0] * u[0] + C[q][1] * u[1] + C[q][2] * u[2]
            cF = C[q][0] * F[0] + C[q][1] * F[1] + C[q][2] * F[2]
            self.f[q] = (self.f[q] * (1 - 1 / c.tau) + _equilibrium(q, rho, *u, usq) / c.tau
                         + guo * WEIGHT[q] * ((cF - uF) * 3 + cu * 9 * cF))
        new = torch.empty_like(self.f)
        for q, (a, b, d) in enumerate(C):
            new[q] = self.f[OPP[q]]
            src = self.f[q]
            if c.compat & PERIODIC_Z:
                src, d = torch.roll(src, d, 0), 0
            to = tuple(slice(max(v, 0), src.shape[i] + min(v, 0)) for i, v in enumerate((d, b, a)))
            fr = tuple(slice(max(-v, 0), src.shape[i] + min(-v, 0)) for i, v in enumerate((d, b, a)))
            new[q][to] = src[fr]
        m = (slice(None), slice(None), slice(1, -1))
        inner = tuple(slice(2, k - 2) for k in (c.nz, c.ny)) + (slice(3, c.nx - 3),)
        rho = sum(new[q][m] for q in range(19))
        self.rho[inner] = rho
        for d in range(3):
            j = sum(C[q][d] * new[q][m] for q in range(19) if C[q][d])
            self.u[d][inner] = (j + 0.5 * F[d][m]) / rho
        for k, p in enumerate(self.pos):
            flat = p.reshape(-1, 3)
            idx, w = self._stencil(flat)
            v = torch.stack([(self.u[d].reshape(-1)[idx] * w).sum(1) for d in range(3)], dim=1).view_as(p)
            if c.compat & PIN_ROW0:
                v[0] = 0.0
            self.pos[k] = p + v
        for q in range(19):
            new[q][:, :, 0] = self.plane[q]
            new[q][:, :, -1] = self.plane[q]
        self.f = new

    def sheet(self, k):
        return torch.cat([self.pos[k], *self.force[k]], dim=-1).cpu()


def _network(widths, p):
    layers, at = [], 0
    for a, b in zip(widths[:-1], widths[1:]):
        layers.append((p[at:at + a * b].view(b, a), p[at + a * b:at + a * b + b]))
        at += a * b + b
    return layers


def _evaluate(layers, X):
    for i, (W, b) in enumerate(layers):
        X = X @ W.T + b
        if i + 1 < len(layers):
            X = torch.nn.functional.gelu(X)
    return X


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    kind = case["kind"]
    if kind == "solver":
        spec, pos = _channel(case, seed)
        flow = _Flow(spec, pos, dev)
        for _ in range(case["steps"]):
            flow.step()
        return {"rho": flow.rho.cpu(), "ux": flow.u[0].cpu(), "uy": flow.u[1].cpu(), "uz": flow.u[2].cpu(),
                "sheets": [flow.sheet(k) for k in range(len(pos))]}
    if kind == "sweep":
        if case["problems"] * case["steps"] > 2500:
            return None
        out = {"codes": None, "sheets": []}
        for k, p in enumerate(_problems(case, seed)):
            s = SheetSpec(p.rows, p.cols, p.width, p.height, p.x0, p.y0, p.z0)
            spec = ChannelSpec(p.nx, p.ny, p.nz, 4, [s], p.tau, p.u_l, p.Ks_l, p.Kb_l, PIN_ROW0)
            r, c = np.meshgrid(np.arange(p.rows), np.arange(p.cols), indexing="ij")
            x = np.stack([np.full(r.shape, p.x0 + p.u_l), p.y0 + p.height / (p.rows - 1) * r,
                          p.z0 + p.width / (p.cols - 1) * c], axis=-1)
            flow = _Flow(spec, [x], dev)
            for _ in range(case["steps"]):
                flow.step()
            out["sheets"].append(flow.sheet(0).reshape(-1))
        out["sheets"] = torch.cat(out["sheets"])
        return out
    w = _widths(case)
    if kind == "train":
        p, X, T = _train_data(case, seed)
        p = torch.from_numpy(p).double().to(dev).requires_grad_(True)
        X, T = (torch.from_numpy(a).double().to(dev).split(case["batch"]) for a in (X, T))
        m, v = torch.zeros_like(p), torch.zeros_like(p)
        for i in range(case["steps"]):
            loss = (_evaluate(_network(w, p), X[i % len(X)]) - T[i % len(T)]).square().mean()
            g, = torch.autograd.grad(loss, p)
            with torch.no_grad():
                m = 0.9 * m + 0.1 * g
                v = 0.999 * v + 0.001 * g * g
                p -= LEARNING_RATE * (m / (1 - 0.9 ** (i + 1))) / ((v / (1 - 0.999 ** (i + 1))).sqrt() + 1e-8)
        return p.detach().cpu()
    rng = np.random.default_rng(seed)
    weights = [torch.from_numpy(_weights(w, rng)).double().to(dev) for _ in range(case["members"])]
    X = torch.from_numpy(rng.uniform(-1, 1, (case["points"], w[0])).astype(np.float32)).double().to(dev)
    return [_evaluate(_network(w, p), X).cpu() for p in weights]
