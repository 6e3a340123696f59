"""The measured work of this framework, through its public entry points.

A program of this framework does four things with it: it solves one spectral
system on its own device arrays (f8_fft_solve), it advances a stored state by
some time steps and takes the new state and the drag history back
(Solver.load / step / store), it does that in FP64 or in FP32-mixed precision,
and it asks for the gradient of the drag (Solver.grad).  The cases are these
uses on the grids of the repository's own workloads (configs.py), from 4 K to
33 M cells, in 2D and 3D, periodic and between walls, with the FFT and the SOR
pressure solver.  Every extent is a power of two (other extents are refused);
the odd sizes are the rows of a wall channel (NY + 2), uneven aspect ratios,
step counts and marker counts.

A case's keys:

    kind       "solve", "run" or "grad"
    flow       "start": the workload's own initial state (C = identity and
               noise, what every run of the benchmark configurations begins
               with); "developed": a flow with vortices of several sizes and a
               stretched conformation tensor, what all later steps work on
    work       the workload that gives Re, Wi, beta, L^2 and dt
    precision  0 FP64, 1 FP32-mixed
    poisson    0 FFT, 1 SOR

What a mixed run computes is single precision (its C, histories and increments
are FP32), so its user takes the snapshot as FP32 tensors; an FP64 run returns
the FP64 arrays that store() fills.
"""
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from fortran8_gb300 import abi, configs, lib
from fortran8_gb300.solver import CylSpec, GridSpec, Solver, State

PI = math.pi
WORK = {"c1_2d": configs.c1_2d, "c2_3d": configs.c2_3d, "c3_channel": configs.c3_channel,
        "c4_adjoint": configs.c4_adjoint, "c5_large": configs.c5_large}
FIELDS = ("u", "v", "w", "p", "c")


def _run(name, work, nx, ny, nz, precision, steps, flow, ncyl, poisson=0, kind="run", every=0):
    return {"name": name, "kind": kind, "work": work, "nx": nx, "ny": ny, "nz": nz, "precision": precision,
            "steps": steps, "flow": flow, "ncyl": ncyl, "poisson": poisson, "checkpoint": every}


def listed():
    return [
        # the smallest call: one pressure solve of a 2D field on the 2D box's grid
        {"name": "solve_2d_128", "kind": "solve", "nx": 128, "ny": 128, "nz": 1, "lhs0": 0.0, "lhs1": -1.0},
        # a viscous solve on the channel's grid, by a program that keeps its own step
        {"name": "solve_256x128x128", "kind": "solve", "nx": 256, "ny": 128, "nz": 128, "lhs0": 1.0, "lhs1": 1.8e-7},
        # the 2D box with one cylinder in FP64: the reference's own 2D run, from its start
        _run("box2d_128_fp64", "c1_2d", 128, 128, 1, 0, 25, "start", 1),
        # a finer 2D flow in the fast precision
        _run("box2d_512_mixed", "c1_2d", 512, 512, 1, 1, 40, "developed", 1),
        # the 3D periodic box in FP64 (the parity configuration), later in its run
        _run("box_64_fp64", "c2_3d", 64, 64, 64, 0, 6, "developed", 1),
        # a channel in FP64: what a user checks a mixed run against
        _run("channel_128x64x64_fp64", "c4_adjoint", 128, 64, 64, 0, 3, "developed", 2),
        # the periodic box in mixed precision, from the workload's start
        _run("box_64_mixed", "c2_3d", 64, 64, 64, 1, 50, "start", 1),
        # the benchmark channel in mixed precision
        _run("channel_256x128x128_mixed", "c3_channel", 256, 128, 128, 1, 40, "developed", 4),
        # the same flow with the SOR pressure solver, on a grid its sweeps are used for
        _run("channel_64x32x32_sor", "c3_channel", 64, 32, 32, 1, 5, "developed", 4, poisson=1),
        # the large channel
        _run("channel_512x256x256_mixed", "c5_large", 512, 256, 256, 1, 12, "developed", 8),
        # the drag gradient of the adjoint channel in mixed precision
        _run("grad_128x64x64_mixed", "c4_adjoint", 128, 64, 64, 1, 40, "developed", 2, kind="grad", every=20),
        # the FP64 gradient on the small grid it is checked on
        _run("grad_32x16x16_fp64", "c4_adjoint", 32, 16, 16, 0, 10, "developed", 2, kind="grad", every=5),
    ]


def draw(rng):
    """One more case of the same ranges (rng: random.Random)."""
    kind = rng.choice(("solve", "run2d", "fp64", "fp64", "mixed", "mixed", "mixed", "sor", "grad"))
    p2 = lambda lo, hi: 1 << rng.randint(lo, hi)
    flow = rng.choice(("start", "developed", "developed"))
    if kind == "solve":
        nx, ny, nz = p2(4, 9), p2(4, 8), rng.choice((1, p2(3, 7)))
        poisson = rng.random() < 0.5
        return {"kind": "solve", "nx": nx, "ny": ny, "nz": nz, "lhs0": 0.0 if poisson else 1.0,
                "lhs1": -1.0 if poisson else 10.0 ** rng.uniform(-7, -4)}
    if kind == "run2d":
        prec, n = rng.randint(0, 1), p2(5, 9)
        c = _run("", "c1_2d", n, n >> rng.randint(0, 1), 1, prec, rng.randint(5, 41), flow, rng.randint(0, 1))
    elif kind == "fp64":
        work = rng.choice(("c2_3d", "c3_channel"))
        nx, ny, nz = p2(5, 7), p2(4, 6), p2(4, 6)
        c = _run("", work, nx, ny, nz, 0, max(1, min(9, (1 << 20) // (nx * ny * nz)) + rng.randint(0, 2)), flow,
                 rng.choice((0, 1, 2)))
    elif kind == "mixed":
        work = rng.choice(("c2_3d", "c3_channel", "c5_large"))
        nx, ny, nz = p2(5, 8), p2(5, 7), p2(4, 7)
        c = _run("", work, nx, ny, nz, 1, rng.randint(7, 45), flow, rng.choice((0, 1, 2, 4)))
    elif kind == "sor":
        c = _run("", rng.choice(("c2_3d", "c3_channel")), p2(5, 6), p2(4, 5), p2(4, 5), rng.randint(0, 1),
                 rng.randint(1, 4), flow, rng.choice((1, 2)), poisson=1)
    else:
        prec = rng.randint(0, 1)
        nx = p2(5, 6) << prec
        n = rng.randint(3, 7) << (2 * prec)
        c = _run("", rng.choice(("c4_adjoint", "c2_3d")), nx, nx >> 1, (nx >> 1) >> rng.randint(0, 1), prec, n, flow,
                 rng.choice((1, 2)), kind="grad", every=rng.choice((0, n // 2 + 1)))
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# inputs

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _generator(seed):
    return np.random.Generator(np.random.PCG64(seed))


def _specs(case):
    """(GridSpec, PhysSpec, cylinders) of a run: square cells of the size that
    the workload's box height gives, the workload's radii and parameters."""
    w = WORK[case["work"]]()
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    h = 2 * PI / ny
    g = GridSpec(w.grid.dim, nx, ny, nz, nx * h, ny * h, nz * h if w.grid.dim == 3 else h, w.grid.bc_y, 0.0)
    n = case["ncyl"]
    r = w.cyls[0].r
    rows = 2 if n >= 4 else 1
    per = max(1, min(n // rows, int(g.lx / (2 * r + 6 * h))))      # as many to a row as fit
    cyls = tuple(CylSpec(g.lx * (2 * a + 1) / (2 * per), g.ly * (2 * b + 1) / (2 * rows), r)
                 for b in range(rows) for a in range(per))[:n]
    return g, w.phys, cyls


def _modes(g, rng, count, kmax, device):
    """Smooth random fields on the cell centres: `count` interior arrays
    (nz, ny, nx) of unit mean square, sums of 4 products of periodic waves."""
    ax = [torch.arange(n, device=device, dtype=torch.float64) * (2 * PI / n) for n in (g.nz, g.ny, g.nx)]
    out = []
    for _ in range(count):
        f = torch.zeros(g.interior_shape, device=device, dtype=torch.float64)
        for _ in range(4):
            k, p = rng.integers(0, kmax + 1, 3), rng.uniform(0, 2 * PI, 3)
            wz, wy, wx = (torch.cos(int(k[q]) * ax[q] + p[q]) for q in range(3))
            f += wz[:, None, None] * wy[None, :, None] * wx[None, None, :]
        out.append(f / f.square().mean().sqrt().clamp_min(1e-3))
    return out


def _fields(case, seed):
    """The initial state's interior values as torch tensors on the device:
    velocity (3), p, C (list of components) and the driving force."""
    g, ph, _ = _specs(case)
    dev, rng = _device(), _generator(seed)
    shape, dim = g.interior_shape, g.dim
    walls = g.bc_y == abi.F8_BC_WALLS
    noise = {"c1_2d": 1e-3, "c2_3d": 1e-3}.get(case["work"], 1e-2)
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(rng.integers(1 << 40)))
    rand = lambda: noise * (torch.rand(shape, generator=gen, device=dev, dtype=torch.float64) - 0.5)
    zero = torch.zeros(shape, device=dev, dtype=torch.float64)
    vel = [zero.clone(), zero.clone(), zero.clone()]
    x, y, z = (torch.arange(1, n + 1, device=dev, dtype=torch.float64) * (l / n)
               for n, l in ((g.nx, g.lx), (g.ny, g.ly), (g.nz, g.lz)))
    hx = g.lx / g.nx
    force = 0.0
    if walls:                                    # Poiseuille profile and its driving force
        half = g.ly / 2
        vel[0] += (1 - ((y - 0.5 * hx - half) / half) ** 2)[None, :, None]
        force = 2.0 / (ph.re * half * half)
    elif dim == 2:
        vel[0] += 1.0
    else:                                        # Taylor-Green in the box's own periods
        sx, sy, sz = 2 * PI / g.lx, 2 * PI / g.ly, 2 * PI / g.lz
        c = lambda a, s, o: torch.cos(s * (a - o * hx))
        vel[0] += torch.sin(sx * x)[None, None, :] * c(y, sy, 0.5)[None, :, None] * c(z, sz, 0.5)[:, None, None]
        vel[1] -= c(x, sx, 0.5)[None, None, :] * torch.sin(sy * y)[None, :, None] * c(z, sz, 0.5)[:, None, None]
    damp = 1.0
    if walls:
        damp = (4 * (y - 0.5 * hx) / g.ly * (1 - (y - 0.5 * hx) / g.ly))[None, :, None]
    for q in range(dim):
        vel[q] += rand()
    p = zero.clone()
    n = dim * (dim + 1) // 2
    diag = {6: (0, 3, 5), 3: (0, 2)}[n]
    conf = [torch.ones_like(zero) if m in diag else zero.clone() for m in range(n)]
    if case["flow"] == "developed":
        for q in range(dim):
            vel[q] += 0.15 * damp * _modes(g, rng, 1, 4, dev)[0]
        p += 0.05 * _modes(g, rng, 1, 4, dev)[0]
        # C = 0.7 I + sum of dyads: symmetric positive definite, tr C up to a
        # few per cent of L^2 in the strained regions
        stretch = math.sqrt(0.01 * ph.lp2)
        pairs = [(a, b) for a in range(dim) for b in range(a, dim)]
        conf = [0.7 * c for c in conf]
        for amp in (stretch, 0.6, 0.3)[:dim]:
            v = _modes(g, rng, dim, 3, dev)
            for m, (a, b) in enumerate(pairs):
                conf[m] += (amp * amp / dim) * v[a] * v[b]
    return g, vel, p, conf, force


def _host(shape, fill=None):
    """A page-locked numpy array (what a program that moves states often keeps)."""
    t = torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    if fill is not None:
        t.fill_(fill)
    return t, t.numpy()


def _state(case, seed):
    """The initial state in page-locked host arrays; histories and Phi are zero
    and left out, as a fresh run leaves them."""
    g, vel, p, conf, force = _fields(case, seed)
    keep, arrays = [], {}

    def put(name, value):
        t, a = _host(value.shape)
        t.copy_(value)
        keep.append(t)
        arrays[name] = a

    pad = lambda f: torch.nn.functional.pad(f, (1, 1, 1, 1, 1, 1))
    for name, f in zip(("u", "v", "w", "p"), vel + [p]):
        put(name, pad(f))
    put("c", torch.stack([pad(f) for f in conf], -1))
    if force:
        put("fx", torch.full(g.interior_shape, force, dtype=torch.float64))
    return State(arrays), keep


class _Solve:
    def __init__(self, case, seed):
        self.case = case
        gen = torch.Generator(device=_device())
        gen.manual_seed(seed)
        shape = (case["nz"], case["ny"], case["nx"])
        self.q = torch.randn(shape, generator=gen, device=_device(), dtype=torch.float64)
        self.phi = torch.empty_like(self.q)
        self.args = (case["nx"], case["ny"], case["nz"]) + tuple(2 * PI / case["ny"] * n for n in
                                                                 (case["nx"], case["ny"], case["nz"]))

    def run(self):
        st = lib.functions()["fft_solve"](*self.args, self.q.data_ptr(), self.phi.data_ptr(), self.case["lhs0"],
                                          self.case["lhs1"])
        if st != abi.F8_OK:
            raise RuntimeError(f"f8_fft_solve: status {st}")
        return self.phi


class _Steps:
    def __init__(self, case, seed):
        self.case = case
        g, ph, cyls = _specs(case)
        self.state, self.keep = _state(case, seed)
        self.solver = Solver(lib.functions(), g, ph, cyls, precision=case["precision"], poisson=case["poisson"])
        if case["kind"] == "run":
            shapes = {n: g.halo_shape for n in FIELDS[:4]}
            shapes["c"] = g.halo_shape + (g.ncomp,)
            self.out_t = {n: _host(s, 0.0)[0] for n, s in shapes.items()}
            self.out = State({n: t.numpy() for n, t in self.out_t.items()})

    def run(self):
        c, s = self.case, self.solver
        s.load(self.state)
        if c["kind"] == "grad":
            _, j, dp, _, drag = s.grad(c["steps"], c["checkpoint"])
            if c["precision"] == abi.F8_MIXED:
                dp, drag, j = dp.astype(np.float32), drag.astype(np.float32), np.float32(j)
            return {"grad": dp, "drag": drag, "objective": j}
        _, drag = s.step(c["steps"])
        s.store(self.out)
        if c["precision"] == abi.F8_MIXED:
            # to the device and to FP32, where the analysis of a snapshot runs
            res = {n: t.to(_device(), non_blocking=True).float() for n, t in self.out_t.items()}
            if drag is not None:
                res["drag"] = drag.astype(np.float32)
        else:
            res = dict(self.out.arrays)
            if drag is not None:
                res["drag"] = drag
        if _specs(c)[0].dim == 2:
            del res["w"]                          # zero in 2D
        return res


def prepare(case, seed):
    return _Solve(case, seed) if case["kind"] == "solve" else _Steps(case, seed)


def run(state):
    return state.run()


def work(case):
    """Bytes and operations that one pass cannot do without: each step reads
    the state once and writes it once (FP64 words of 8 bytes, FP32 of 4; U, V,
    W, P are carried to more than FP32 in both precisions), with the transforms
    and stencils of the model; a gradient is a forward step that keeps its
    fields and a reverse step of twice its operations."""
    n = case["nx"] * case["ny"] * case["nz"]
    lg = math.log2(case["nx"] * case["ny"] * case["nz"])
    if case["kind"] == "solve":
        return {"bytes": 16.0 * n, "flops": 5.0 * n * lg}
    dim = 2 if case["nz"] == 1 else 3
    comps, word = dim * (dim + 1) // 2, 8 if case["precision"] == 0 else 4
    per_step = 2 * ((dim + 1) * 8 + (comps + 2 * dim) * word)      # U..P, C, the two histories
    flops = (dim + 1) * 5.0 * lg + (2000.0 if dim == 3 else 500.0)
    through_host = 0.0 if case["kind"] == "grad" else 8.0 * (dim + 1 + comps)
    if case["kind"] == "grad":
        per_step, flops = 3 * per_step, 3 * flops
    return {"bytes": n * (per_step * case["steps"] + 8.0 * (dim + 1 + comps) + through_host),
            "flops": n * flops * case["steps"]}


# ---------------------------------------------------------------------------
# the same results in 64 bits, in plain torch: the discrete equations written
# once for 2D and 3D, differentiable (for the gradient cases)

class _Model:
    """The discrete SMAC + FENE-P + direct-forcing step in torch FP64."""

    def __init__(self, case, device):
        self.g, self.ph, self.cyls = _specs(case)
        g = self.g
        self.dim, self.dev = g.dim, device
        self.n = (g.nx, g.ny, g.nz)
        h = g.ly / g.ny
        self.h = (g.lx / g.nx, h, g.lz / g.nz if g.dim == 3 else h)
        self.walls = g.bc_y == abi.F8_BC_WALLS
        self.sor = case["poisson"] == abi.F8_POISSON_SOR
        self.pairs = [(a, b) for a in range(self.dim) for b in range(a, self.dim)]
        self.lookup = {}
        for m, (a, b) in enumerate(self.pairs):
            self.lookup[a, b] = self.lookup[b, a] = m
        self.markers = self._marker_list()

    # -- arrays: interior (nz, rows, nx), with ghosts (nz+2, rows+2, nx+2) ----
    def wrap(self, a, rows=None):
        """Periodic ghosts in x and z, and in y when there are no walls; with
        walls the given ghost rows (lo, hi), each (nz, 1, nx)."""
        a = torch.cat([a[:, -1:], a, a[:, :1]], 1) if rows is None else torch.cat([rows[0], a, rows[1]], 1)
        a = torch.cat([a[:, :, -1:], a, a[:, :, :1]], 2)
        return torch.cat([a[-1:], a, a[:1]], 0)

    def ghosts(self, a, kind):
        if not self.walls:
            return self.wrap(a)
        lo, hi = a[:, :1], a[:, -1:]
        if kind in (0, 2):
            lo, hi = -lo, 2 * self.g.uwall * (kind == 0) - hi
        elif kind == 1:
            a = torch.cat([a[:, :-1], torch.zeros_like(hi)], 1)
            lo = hi = torch.zeros_like(hi)
        elif kind == "c":
            lo, hi = 2 * lo - a[:, 1:2], 2 * hi - a[:, -2:-1]
        return self.wrap(a, (lo, hi))

    @staticmethod
    def at(a, off=(0, 0, 0)):
        i, j, k = off
        nz, ny, nx = (s - 2 for s in a.shape)
        return a[1 + k:1 + k + nz, 1 + j:1 + j + ny, 1 + i:1 + i + nx]

    def shift(self, d, s=1):
        return tuple(s if q == d else 0 for q in range(3))

    def add(self, *offs):
        return tuple(sum(o[q] for o in offs) for q in range(3))

    # -- polymer ---------------------------------------------------------------
    def least_eigenvalue(self, a):
        if self.dim == 2:
            s = torch.sqrt((a[0] - a[2]) ** 2 + 4 * a[1] ** 2)
            return (a[0] + a[2] - s) / 2
        a2 = -(a[0] + a[3] + a[5])
        a1 = a[0] * a[3] + a[3] * a[5] + a[5] * a[0] - a[4] ** 2 - a[2] ** 2 - a[1] ** 2
        a0 = -(a[0] * a[3] * a[5] + 2 * a[1] * a[4] * a[2] - a[0] * a[4] ** 2 - a[1] ** 2 * a[5] - a[2] * a[3] * a[2])
        p = a1 - a2 * a2 / 3
        q = a0 - a1 * a2 / 3 + 2 * a2 ** 3 / 27
        t = (q / 2) ** 2 + (p / 3) ** 3
        lam = 2 * torch.sqrt(-p / 3) * torch.cos(torch.acos(3 * q / (2 * p) * torch.sqrt(-3 / p)) / 3 + 2 * PI / 3) - a2 / 3
        return torch.where(t >= 0, torch.full_like(lam, -100.0), lam)     # the model's value for equal roots

    FACE = ((0.0, 1.5, -0.5), (0.5, 0.5, 0.0), (0.25, 1.0, -0.25), (0.0, 1.0, 0.0))

    def choose(self, cm, c0, cp):
        with torch.no_grad():
            best = torch.zeros_like(c0[0])
            code = torch.full_like(c0[0], 3, dtype=torch.long)
            for l in range(3):
                w = self.FACE[l]
                lo = self.least_eigenvalue([w[0] * m + w[1] * c + w[2] * p for m, c, p in zip(cm, c0, cp)])
                hi = self.least_eigenvalue([-w[0] * m + (1 + w[0] + w[2]) * c - w[2] * p for m, c, p in zip(cm, c0, cp)])
                v = torch.fmin(lo, hi)
                # 3D: the first largest of the three and 0; 2D: the last that is not below the best so far
                better = (v >= best) if self.dim == 2 else ((v > best) | ((v == 0) & (best == 0) & (code == 3)))
                best, code = torch.where(better, v, best), torch.where(better, torch.full_like(code, l), code)
            return code

    def polymer(self, conf, vel, wi, lp2):
        """C of the next step on the updated rows (with walls the ghost rows too,
        outside of which C and the velocity are zero)."""
        dt, dim = self.ph.dt, self.dim
        if self.walls:
            grow = lambda a: torch.nn.functional.pad(a, (0, 0, 1, 1))
            conf, vel = [grow(c) for c in conf], [grow(v) for v in vel]
        c0 = [self.at(c) for c in conf]
        b = [torch.zeros_like(c) for c in c0]
        for d in range(dim):
            cm = [self.at(c, self.shift(d, -1)) for c in conf]
            cp = [self.at(c, self.shift(d, 1)) for c in conf]
            code = self.choose(cm, c0, cp)
            w = torch.tensor(self.FACE, dtype=torch.float64, device=self.dev)[code]
            w0, w2 = w[..., 0], w[..., 2]
            v1, v2 = self.at(vel[d], self.shift(d, -1)), self.at(vel[d])
            r = dt / (2 * self.h[d])
            sm, sp = 0.5 / dim + (v1 - v1.abs()) * r, 0.5 / dim + (-v2 - v2.abs()) * r
            tm, tp = (v1 + v1.abs()) * r, (-v2 + v2.abs()) * r
            axis = {0: 2, 1: 1, 2: 0}[d]

            def step_to(f, s, axis=axis, d=d):
                if d == 1 and self.walls:
                    f = torch.roll(f, -s, axis)
                    edge = torch.zeros_like(f[:, :1])
                    return torch.cat([f[:, :-1], edge], 1) if s > 0 else torch.cat([edge, f[:, 1:]], 1)
                return torch.roll(f, -s, axis)

            for m in range(len(b)):
                plus = w0 * cm[m] + (1 - w0 - w2) * c0[m] + w2 * cp[m]
                minus = -w0 * cm[m] + (1 + w0 + w2) * c0[m] - w2 * cp[m]
                b[m] = b[m] + sm * plus + sp * minus + tp * step_to(plus, 1) + tm * step_to(minus, -1)
        for a in range(dim):
            b[self.lookup[a, a]] = b[self.lookup[a, a]] + dt / wi
        # A = -dt (velocity gradient)^T at the cell, first index the component
        A = [[None] * dim for _ in range(dim)]
        for a in range(dim):
            for e in range(dim):
                if a == e:
                    grad = (self.at(vel[a]) - self.at(vel[a], self.shift(a, -1))) / self.h[a]
                else:
                    grad = sum(self.at(vel[a], self.add(self.shift(a, o), self.shift(e, 1)))
                               - self.at(vel[a], self.add(self.shift(a, o), self.shift(e, -1))) for o in (-1, 0)) / (4 * self.h[e])
                A[a][e] = -dt * grad
        return self.lyapunov(A, b, [c.detach() for c in c0], wi, lp2)

    def residual(self, A, b, x, wi, lp2):
        tr = sum(x[self.lookup[a, a]] for a in range(self.dim))
        f = (lp2 - self.dim) / (lp2 - tr)
        res = []
        for m, (a, e) in enumerate(self.pairs):
            s = (1 + f * self.ph.dt / wi) * x[m] - b[m]
            for k in range(self.dim):
                s = s + A[a][k] * x[self.lookup[k, e]] + x[self.lookup[a, k]] * A[e][k]
            res.append(s)
        return res

    def correction(self, A, x, res, wi, lp2):
        """J^-1 res with the exact Jacobian at x (elimination, cell by cell)."""
        n, dt = len(x), self.ph.dt
        diag = [self.lookup[a, a] for a in range(self.dim)]
        tr = sum(x[m] for m in diag)
        f, fp = (lp2 - self.dim) / (lp2 - tr), (lp2 - self.dim) / (lp2 - tr) ** 2
        zero = torch.zeros_like(x[0])
        J = [[zero for _ in range(n)] for _ in range(n)]
        for m, (a, e) in enumerate(self.pairs):
            J[m][m] = J[m][m] + 1 + f * dt / wi
            for k in range(self.dim):
                J[m][self.lookup[k, e]] = J[m][self.lookup[k, e]] + A[a][k]
                J[m][self.lookup[a, k]] = J[m][self.lookup[a, k]] + A[e][k]
            for q in diag:
                J[m][q] = J[m][q] + fp * dt / wi * x[m]
        r = list(res)
        for k in range(n):
            inv = 1 / J[k][k]
            J[k] = [v * inv for v in J[k]]
            r[k] = r[k] * inv
            for m in range(n):
                if m != k:
                    fac = J[m][k]
                    J[m] = [J[m][q] - fac * J[k][q] if q > k else J[m][q] for q in range(n)]
                    r[m] = r[m] - fac * r[k]
        return r

    def lyapunov(self, A, b, x, wi, lp2):
        num = lambda v: v.detach() if torch.is_tensor(v) else v
        wn, ln = num(wi), num(lp2)
        with torch.no_grad():
            Ad, bd = [[v.detach() for v in row] for row in A], [v.detach() for v in b]
            for _ in range(5):
                x = [a - d for a, d in zip(x, self.correction(Ad, x, self.residual(Ad, bd, x, wn, ln), wn, ln))]
        if not any(v.requires_grad for v in b + [v for row in A for v in row]):
            return x
        # the implicit-function derivative: one more step whose matrix is held
        res = self.residual(A, b, x, wi, lp2)
        return [a - d for a, d in zip(x, self.correction(Ad, x, res, wn, ln))]

    def stress(self, conf, wi, beta, lp2):
        tr = sum(conf[self.lookup[a, a]] for a in range(self.dim))
        f = (lp2 - self.dim) / (lp2 - tr)
        s = {k: f * conf[m] - (1.0 if k[0] == k[1] else 0.0) for m, k in enumerate(self.pairs)}
        out = []
        for a in range(self.dim):
            t = 0
            for e in range(self.dim):
                c = s[min(a, e), max(a, e)]
                if a == e:
                    t = t + (self.at(c, self.shift(a)) - self.at(c)) / self.h[a]
                else:
                    t = t + sum(self.at(c, self.add(self.shift(a, o), self.shift(e, 1)))
                                - self.at(c, self.add(self.shift(a, o), self.shift(e, -1))) for o in (0, 1)) / (4 * self.h[e])
            out.append((1 - beta) / (self.ph.re * wi) * t)
        return out

    def advect_diffuse(self, vel, beta):
        conv, visc = [], []
        for a in range(self.dim):
            c = l = 0
            for e in range(self.dim):
                he = self.h[e]
                if a == e:
                    lo = (self.at(vel[a], self.shift(a, -1)) + self.at(vel[a])) / 2
                    hi = (self.at(vel[a], self.shift(a)) + self.at(vel[a])) / 2
                    c = c + (hi * hi - lo * lo) / he
                else:
                    flux = [(self.at(vel[e], self.shift(e, o)) + self.at(vel[e], self.add(self.shift(a), self.shift(e, o)))) / 2
                            * (self.at(vel[a], self.shift(e, o)) + self.at(vel[a], self.shift(e, o + 1))) / 2 for o in (-1, 0)]
                    c = c + (flux[1] - flux[0]) / he
                l = l + (self.at(vel[a], self.shift(e, -1)) - 2 * self.at(vel[a]) + self.at(vel[a], self.shift(e))) / (he * he)
            conv.append(-c)
            visc.append(beta / self.ph.re * l)
        return conv, visc

    # -- solves ----------------------------------------------------------------
    def waves(self, d, half=False):
        n = self.n[d]
        m = torch.arange(n // 2 + 1 if half else n, device=self.dev, dtype=torch.float64)
        return 2 * (1 - torch.cos(m * (2 * PI / n))) / self.h[d] ** 2

    def periodic(self, q, lhs0, lhs1):
        dims = (0, 1, 2)
        lam = self.waves(0, True)[None, None, :] + self.waves(1)[None, :, None]
        if self.dim == 3:
            lam = lam + self.waves(2)[:, None, None]
        lhs = lhs0 + lhs1 * lam
        zero = lhs.detach().abs() < 1e-16
        spec = torch.fft.rfftn(q, dim=dims)
        spec = torch.where(zero, torch.zeros_like(spec), spec / torch.where(zero, torch.ones_like(lhs), lhs))
        return torch.fft.irfftn(spec, s=q.shape, dim=dims)

    def between_walls(self, q, kind, kap):
        """Rows 0..NY+1 of the tridiagonal systems of the (kx, kz) modes, by the
        Thomas recurrence (its zero-pivot guard pins the mean pressure mode)."""
        ny, iy2 = self.n[1], 1 / self.h[1] ** 2
        spec = torch.fft.fft(torch.fft.rfft(q, dim=2), dim=0)
        lam = self.waves(2)[:, None] + self.waves(0, True)[None, :] if self.dim == 3 else self.waves(0, True)[None, :]
        one, zero = torch.ones_like(lam), torch.zeros_like(lam)
        none = torch.zeros_like(spec[:, 0])
        end = {0: 1.0, 2: 1.0, 1: 0.0, "p": -1.0}[kind]
        rows, last = [], ny + 1
        for j in range(ny + 2):
            inside = 1 <= j <= ny and not (kind == 1 and j == ny)
            if not inside:
                low, up = (end if j == last else 0.0), (end if j == 0 else 0.0)
                a, below, above, rhs = one, low, up, none
                if kind == 0 and j == last and self.g.uwall:
                    rhs = none.clone()
                    rhs[0, 0] = 2 * self.g.uwall * self.n[0] * self.n[2]
            else:
                c = iy2 if kind == "p" else -kap * iy2
                a = -(lam + 2 * iy2) if kind == "p" else 1 + kap * (lam + 2 * iy2)
                below = above = c
                rhs = spec[:, j - 1]
            if j == 0:
                p, y = -above * one, rhs
            else:
                den = a + below * p
                small = den.detach().abs() < 1e-16
                inv = 1 / torch.where(small, one, den)
                y = torch.where(small, none, (rhs - below * y) * inv)
                p = torch.where(small, zero, -above * inv)
            rows.append((p, y))
        x = rows[-1][1]
        sol = [x]
        for p, y in rows[-2::-1]:
            x = p * x + y
            sol.append(x)
        full = torch.stack(sol[::-1], 1)
        return torch.fft.irfft(torch.fft.ifft(full, dim=0), n=self.n[0], dim=2)

    def viscous_solve(self, q, comp, kap):
        if not self.walls:
            return self.ghosts(self.periodic(q, 1.0, kap), comp)
        return self.ghosts(self.between_walls(q, comp, kap)[:, 1:-1], comp)

    def pressure_solve(self, q):
        phi = self.periodic(q, 0.0, -1.0) if not self.walls else self.between_walls(q, "p", 0.0)[:, 1:-1]
        if self.sor:
            phi = phi - phi.mean()
        return self.ghosts(phi, "p")

    # -- immersed cylinders ------------------------------------------------------
    def _marker_list(self):
        """(cylinder, offset from its centre) of the markers of filled cylinders:
        concentric shells one cell apart, about one marker per cell."""
        out, h = [], self.h[0]
        for l, cy in enumerate(self.cyls):
            dc = 2 * cy.r
            laps = int(dc / (2 * h))
            counts = [int(math.floor(PI * (dc - 2 * i * h) / h + 0.5)) for i in range(laps + 1)]
            counts[laps] = counts[laps] or 1
            for i, n in enumerate(counts):
                rad = (dc - 2 * i * h) / 2
                out += [(l, rad * math.cos(2 * PI / n * j), rad * math.sin(2 * PI / n * j)) for j in range(1, n + 1)]
        return out

    def forces(self, ua, centres):
        """Direct forcing of resting cylinders: the interior force fields and
        the drag (cylinder, component), with Roma's three-point kernel."""
        dt, dim, h = self.ph.dt, self.dim, self.h
        cyl = torch.tensor([m[0] for m in self.markers], device=self.dev)
        off = torch.tensor([m[1:] for m in self.markers], device=self.dev, dtype=torch.float64)
        pos = centres[cyl] + off
        nz, ny, nx = ua[0].shape
        three = torch.arange(3, device=self.dev)

        def roma(r):
            a = r.abs()
            inner, outer = a < 0.5, (a >= 0.5) & (a < 1.5)
            safe = lambda v, on: torch.sqrt(torch.where(on, v, torch.ones_like(v)))
            return torch.where(inner, (1 + safe(1 - 3 * r * r, inner)) / 3,
                               torch.where(outer, (5 - 3 * a - safe(1 - 3 * (1 - a) ** 2, outer)) / 6, torch.zeros_like(r)))

        planes = torch.arange(1, self.n[2] + 1, device=self.dev)
        fields, drags = [], []
        for c in range(dim):
            idx, wt = [], []
            for d in range(2):
                first = torch.trunc(pos[:, d].detach() / h[d] - (0.5 if d == c else 0.0)).long()
                ii = first[:, None] + three
                grid = (ii.double() - 0.5 + (0.5 if d == c else 0.0)) * h[d]
                idx.append(ii)
                wt.append(roma((grid - pos[:, d:d + 1]) / h[d]))
            if dim == 3:
                kk = planes[:, None] + three - 1
                zz = (kk.double() - 0.5 + (0.5 if c == 2 else 0.0)) * h[2]
                wz = roma((zz - (planes.double() - 0.25)[:, None] * h[2]) / h[2])
            else:
                kk, wz = planes[:, None], torch.ones((1, 1), device=self.dev, dtype=torch.float64)
            wgt = wz[:, None, :, None, None] * wt[1][None, :, None, :, None] * wt[0][None, :, None, None, :]
            flat = (kk[:, None, :, None, None] * ny + idx[1][None, :, None, :, None]) * nx + idx[0][None, :, None, None, :]
            force = -(ua[c].reshape(-1)[flat] * wgt).sum((2, 3, 4)) / dt                 # (planes, markers)
            drag = -torch.zeros(len(self.cyls), device=self.dev, dtype=torch.float64).index_add(0, cyl, force.sum(0))
            drags.append(drag * math.prod(h[:dim]))
            full = torch.zeros(nz * ny * nx, device=self.dev, dtype=torch.float64).index_add(
                0, flat.reshape(-1), (force[:, :, None, None, None] * wgt).reshape(-1)).reshape(nz, ny, nx)
            # what lands on the ghosts belongs to the periodic images
            full = torch.cat([full[:, :, 1:2] + full[:, :, -1:], full[:, :, 2:-2], full[:, :, -2:-1] + full[:, :, :1]], 2)
            if not self.walls:
                full = torch.cat([full[:, 1:2] + full[:, -1:], full[:, 2:-2], full[:, -2:-1] + full[:, :1]], 1)
            else:
                full = full[:, 1:-1]
            if dim == 3:
                full = torch.cat([full[1:2] + full[-1:], full[2:-2], full[-2:-1] + full[:1]], 0)
            else:
                full = full[1:-1]
            fields.append(full)
        while len(drags) < 3:
            drags.append(torch.zeros_like(drags[0]))
        return fields, torch.stack(drags, 1)

    # -- one step -----------------------------------------------------------------
    def step(self, s, prm, first):
        dt, dim, re = self.ph.dt, self.dim, self.ph.re
        wi, beta, lp2, centres = prm
        conf = self.polymer(s["c"], s["vel"], wi, lp2)
        if self.walls:      # rows 0..NY+1 are updated; periodic ghosts in x and z
            full = [self.wrap(c[:, 1:-1], (c[:, :1], c[:, -1:])) for c in conf]
        else:
            full = [self.wrap(c) for c in conf]
        T = self.stress(full, wi, beta, lp2)
        A, B = self.advect_diffuse(s["vel"], beta)
        A0, T0 = (A, T) if first else (s["A"], s["T"])
        ua = []
        for c in range(dim):
            gp = -(self.at(s["p"], self.shift(c)) - self.at(s["p"])) / self.h[c]
            f = s["force"] if c == 0 else 0.0
            ua.append(self.at(s["vel"][c]) + dt * (gp + (3 * A[c] - A0[c]) / 2 + B[c] + (T[c] + T0[c]) / 2 + f))
        drag, force = None, [0.0] * dim
        if self.cyls:
            force, drag = self.forces([self.ghosts(u, c) for c, u in enumerate(ua)], centres)
        kap = dt * beta / re / 2
        up = [self.viscous_solve(ua[c] + dt * force[c] - dt * B[c] / 2, c, kap) for c in range(dim)]
        div = sum((self.at(up[c]) - self.at(up[c], self.shift(c, -1))) / self.h[c] for c in range(dim)) / dt
        phi = self.pressure_solve(div)
        vel = [self.ghosts(self.at(up[c]) - dt * (self.at(phi, self.shift(c)) - self.at(phi)) / self.h[c], c)
               for c in range(dim)]
        lap = sum((self.at(phi, self.shift(c, -1)) - 2 * self.at(phi) + self.at(phi, self.shift(c))) / self.h[c] ** 2
                  for c in range(dim))
        p = self.ghosts(self.at(s["p"]) + self.at(phi) - kap * lap, "p")
        if self.walls:      # the ghost rows of C are extrapolated at the end of the step
            full = [self.ghosts(c[:, 1:-1], "c") for c in conf]
        return {"vel": vel, "p": p, "c": full, "A": A, "T": T, "force": s["force"]}, drag

    def start(self, case, seed):
        _, vel, p, conf, force = _fields(case, seed)
        return {"vel": [self.ghosts(v, c) for c, v in enumerate(vel)][:self.dim], "p": self.ghosts(p, "p"),
                "c": [self.ghosts(c, "c") for c in conf], "A": None, "T": None, "force": force}


def _exact_run(case, seed):
    m = _Model(case, _device())
    prm = (m.ph.wi, m.ph.beta, m.ph.lp2,
           torch.tensor([[c.xc, c.yc] for c in m.cyls], device=m.dev, dtype=torch.float64))
    drags = []
    with torch.no_grad():
        s = m.start(case, seed)
        for n in range(case["steps"]):
            s, d = m.step(s, prm, n == 0)
            drags.append(d)
    res = dict(zip(("u", "v", "w"), s["vel"]))
    res["p"], res["c"] = s["p"], torch.stack(s["c"], -1)
    if m.dim == 2:         # the ghost planes of a 2D field are copies
        res = {n: torch.cat([v[1:2]] * 3) for n, v in res.items()}
    if m.cyls:
        res["drag"] = torch.stack(drags)
    return res


def _exact_grad(case, seed):
    m = _Model(case, _device())
    leaf = lambda v: torch.tensor(v, device=m.dev, dtype=torch.float64, requires_grad=True)
    prm = (leaf(m.ph.wi), leaf(m.ph.beta), leaf(m.ph.lp2), leaf([[c.xc, c.yc] for c in m.cyls]))
    s, drags = m.start(case, seed), []
    for n in range(case["steps"]):
        s, d = checkpoint(m.step, s, prm, n == 0, use_reentrant=False)
        drags.append(d)
    drag = torch.stack(drags)
    j = drag[:, :, 0].sum() / case["steps"]
    j.backward()
    grad = torch.cat([torch.stack([prm[q].grad for q in range(3)]), prm[3].grad.reshape(-1)])
    return {"grad": grad, "drag": drag.detach(), "objective": j.item()}


def exact(case, seed):
    if case["kind"] == "solve":
        s = _Solve(case, seed)
        m = _Model(_run("", "c2_3d", case["nx"], case["ny"], max(case["nz"], 4), 0, 1, "start", 0), _device())
        m.n, m.dim = (case["nx"], case["ny"], case["nz"]), 3
        return m.periodic(s.q, case["lhs0"], case["lhs1"])
    return _exact_grad(case, seed) if case["kind"] == "grad" else _exact_run(case, seed)
