"""Timed workloads of the immersed-boundary time step, through its public API.

A pass advances a case by ``steps`` time steps (one ``IBMSolver.iterate``
call, or one ``Batch.iterate`` call for an ensemble) from wherever the last
pass left it and reads u, v, w and p back to pinned host memory, as a
program does that marches a flow and keeps snapshots.  The solver (grid,
body, boundary conditions, multigrid, recorded step graphs) is what such a
program keeps between passes; the seed makes the initial velocity.

Two kinds of run:

* ``fp64``: the reference's own arithmetic in verification runs, both solves
  to 1e-14 (the parity tests' 1e-12 and the digits that the pressure of a
  closed domain loses).  Snapshots are FP64.
* ``mixed32``, ``mixed`` and ``mixed_mg``: production runs, momentum to
  1e-6 as in the benchmark and the job server and max|div U| <= 1e-9 (their
  1e-8 bound with a digit to spare).  Snapshots keep the digits that these
  stopping tests determine: velocity in FP32, as the reference's result file
  stores it, and p in half precision.
"""
import importlib
import math

import numpy as np
import torch

ibm = importlib.import_module("2020researchproject_gb300")
geometry = importlib.import_module("2020researchproject_gb300.geometry")
workloads = importlib.import_module("2020researchproject_gb300.workloads")

FIELDS = ("u1", "u2", "u3", "p")
MODES = {"fp64": "FP64", "mixed": "MIXED", "mixed_mg": "MIXED_MG", "mixed32": "MIXED32"}


def _case(name, flow, nx, ny, nz, mode, steps, re, members=0, grids=0):
    return dict(name=name, flow=flow, nx=nx, ny=ny, nz=nz, mode=mode, steps=steps, re=re, members=members, grids=grids)


def listed():
    return [
        # The smallest served job: a 32^3 lid-driven cavity, bound by launches.
        _case("cavity32_mixed32", "cavity", 32, 32, 32, "mixed32", 20, 400.0),
        # The reference's cavity driver (64^3, Re 1000) in its own arithmetic.
        _case("cavity64_fp64", "cavity", 64, 64, 64, "fp64", 4, 1000.0),
        # The same grid in production settings.
        _case("cavity64_mixed32", "cavity", 64, 64, 64, "mixed32", 20, 1000.0),
        # A long, ragged served cavity in the job server's default mode.
        _case("cavity213x32x59_mixed", "cavity", 213, 32, 59, "mixed", 10, 797.0),
        # Flow past a sphere at the benchmark's size: verification run ...
        _case("sphere192_fp64", "sphere", 192, 128, 128, "fp64", 2, 300.0),
        # ... and the headline production run.
        _case("sphere192_mixed32", "sphere", 192, 128, 128, "mixed32", 20, 300.0),
        # The largest served job: a uniform 256x128x128 grid around a sphere.
        _case("sphere256_mixed32", "obstacle", 256, 128, 128, "mixed32", 15, 550.0),
        # Turbulent channel LES, periodic in two axes, at the benchmark's size.
        _case("channel128_mixed32", "channel", 128, 96, 128, "mixed32", 8, 16200.0),
        # A small channel in the reference's arithmetic, odd across the walls.
        _case("channel48_fp64", "channel", 48, 37, 40, "fp64", 4, 16200.0),
        # A cluster of boxes on a ragged grid, as the sweeps over geometry run it.
        _case("boxes95x61x47_mixed32", "boxes", 95, 61, 47, "mixed32", 20, 240.0),
        # The same kind of body in the reference's arithmetic.
        _case("boxes64x48x40_fp64", "boxes", 64, 48, 40, "fp64", 4, 240.0),
        # Twelve uneven immersed-body cases advanced together by one batch.
        _case("ensemble12_mixed32", "ensemble", 96, 64, 64, "mixed32", 20, 0.0, members=12, grids=2024),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same ranges: grids from 32 to 256x128x128 with any
    parity, Re 100-1000 (the channel's 16200), every flow and mode."""
    flow = rng.choice(["cavity", "cavity", "sphere", "obstacle", "boxes", "channel", "ensemble"])
    mode = rng.choice(["mixed32", "mixed32", "mixed32", "fp64", "mixed", "mixed_mg"])
    if flow == "ensemble":
        return _case("drawn", flow, 96, 64, 64, "mixed32" if mode == "fp64" else mode, rng.randint(5, 20), 0.0,
                     members=rng.randint(3, 12), grids=rng.randint(1, 1 << 30))
    nx, ny, nz = _log_int(rng, 32, 256), _log_int(rng, 32, 128), _log_int(rng, 32, 128)
    budget = 4_000_000 if mode == "fp64" else 40_000_000   # cell-steps of the largest listed cases, at most
    steps = max(1, min(20, budget // (nx * ny * nz)))
    re = 16200.0 if flow == "channel" else round(rng.uniform(100.0, 1000.0), 3)
    return _case("drawn", flow, nx, ny, nz, mode, steps, re, grids=rng.randint(1, 1 << 30))


def _flow(case):
    """The workload description (faces, Re, dt, boundary conditions, body)."""
    nx, ny, nz, re = case["nx"], case["ny"], case["nz"], case["re"]
    if case["flow"] == "cavity":
        n = max(nx, ny, nz)
        return dict(xf=geometry.uniform_faces(0.0, 1.0, nx), yf=geometry.uniform_faces(0.0, 1.0, ny),
                    zf=geometry.uniform_faces(0.0, 1.0, nz), re=re, dt=0.064 / n,
                    bc=["W wall", "E wall", "S wall", "N wall", "D wall", "U vel 1 0 0"], init=(0.0, 0.0, 0.0, 0.0))
    if case["flow"] == "sphere":
        return workloads.sphere(nx, ny, nz, Re=re, dt=5e-3 * 128.0 / max(ny, nz), subdivisions=5 if nx > 128 else 4)
    if case["flow"] == "channel":
        return workloads.channel(nx, ny, nz, Re=re)
    # Uniform grid on [-4, 8] x [-3, 3]^2 around a sphere or a cluster of boxes.
    h = min(12.0 / nx, 6.0 / ny, 6.0 / nz)
    if case["flow"] == "obstacle":
        stl = workloads.icosphere_stl(3, 0.5)
    else:
        rng = np.random.Generator(np.random.Philox(case["grids"] + 11))
        boxes = workloads._boxes(rng, int(rng.integers(1, 5)))
        stl = workloads._body_stl("boxes", dict(boxes=boxes), ("boxes", tuple(boxes)))
    return dict(xf=geometry.uniform_faces(-4.0, 8.0, nx), yf=geometry.uniform_faces(-3.0, 3.0, ny),
                zf=geometry.uniform_faces(-3.0, 3.0, nz), re=re, dt=0.25 * h,
                bc=["W vel 1 0 0", "E press 0", "S slip", "N slip", "D slip", "U slip"], stl=stl,
                init=(1.0, 0.0, 0.0, 0.0))


def _flows(case):
    if case["flow"] == "ensemble":
        return workloads.ensemble(case["members"], seed=case["grids"])
    return [_flow(case)]


def _tols(case):
    """(relative tolerance of the solves, bound on max|div U|; 0: none)."""
    if case["mode"] == "fp64":
        return 1e-14, 0.0
    return 1e-6, 1e-9


def _padded(centres):
    return np.concatenate([centres[:1]] * 2 + [centres] + [centres[-1:]] * 2)


def _initial(flow, seed):
    """Initial (u1, u2, u3, p): the workload's state plus a seeded smooth
    disturbance of a few per cent (the channel: its own 10% noise)."""
    if flow.get("init") == "poiseuille":
        return workloads.initial_state(flow, seed)
    state = [np.array(a) for a in workloads.initial_state(flow)]
    rng = np.random.default_rng(seed)
    s = [2.0 * np.pi * (_padded((f[1:] + f[:-1]) / 2) - f[0]) / (f[-1] - f[0])
         for f in (np.asarray(flow[k]) for k in ("xf", "yf", "zf"))]
    for l in range(3):
        for _ in range(3):
            m, ph = rng.integers(1, 4, size=3), rng.uniform(0, 2 * np.pi, size=3)
            w = [np.sin(m[a] * s[a] + ph[a]) for a in range(3)]
            state[l] += 0.02 * rng.uniform(-1, 1) * w[0][:, None, None] * w[1][None, :, None] * w[2][None, None, :]
    return state


def prepare(case, seed):
    flows = _flows(case)
    solvers, host, out = [], [], []
    tol, div_tol = _tols(case)
    for q, flow in enumerate(flows):
        s = workloads.build_solver(ibm, flow, tol=tol, div_tol=div_tol)
        s.set_precision(getattr(ibm, MODES[case["mode"]]))
        s.init_flow_array(*_initial(flow, seed + 1000 * q))
        solvers.append(s)
        shape = tuple(n + 4 for n in s.shape)
        fields = [torch.zeros(shape, dtype=torch.float64, pin_memory=True) for _ in FIELDS]
        host.append([f.numpy() for f in fields])
        out.append(fields if case["mode"] == "fp64" else
                   [torch.zeros(shape, dtype=torch.float16 if f == "p" else torch.float32) for f in FIELDS])
    batch = ibm.Batch(solvers) if case["flow"] == "ensemble" else None
    return dict(case=case, solvers=solvers, host=host, out=out, batch=batch)


def run(state):
    case = state["case"]
    if state["batch"] is not None:
        state["batch"].iterate(case["steps"])
    else:
        state["solvers"][0].iterate(case["steps"])
    for s, host, out in zip(state["solvers"], state["host"], state["out"]):
        for name, h, o in zip(FIELDS, host, out):
            s.get_field_into(name, h)
            if o.dtype != torch.float64:
                o.copy_(torch.from_numpy(h))
    return state["out"]


def work(case):
    """Of one step, per cell: u, U, p and N of the last step read and their
    new values written (10 doubles each way) and the flags read; the
    stencils of convection, both right-hand sides, one application of the
    momentum and pressure operators each and the projection, about 400
    operations; then the snapshot's four fields."""
    cells = sum((len(f["xf"]) + 3) * (len(f["yf"]) + 3) * (len(f["zf"]) + 3) for f in _flows(case))
    return {"bytes": cells * (161.0 * case["steps"] + 64.0), "flops": cells * 400.0 * case["steps"]}


# ------------------------------------------------------------------ exact --
class _Axis:
    """Widths, centres and Crank-Nicolson coefficients of one axis, padded
    by two cells on each side (mirrored widths, or wrapped ones)."""

    def __init__(self, faces, periodic, c, dev):
        d = np.diff(np.asarray(faces, dtype=np.float64))
        self.n, self.periodic = len(d), periodic
        low, high = (d[-2:], d[:2]) if periodic else (d[1::-1], d[:-3:-1])
        d = np.concatenate([low, d, high])
        x = np.empty(self.n + 4)
        x[2:-2] = (np.asarray(faces)[1:] + np.asarray(faces)[:-1]) / 2
        for q in (1, 0):
            x[q] = x[q + 1] - (d[q] + d[q + 1]) / 2
        for q in (self.n + 2, self.n + 3):
            x[q] = x[q - 1] + (d[q] + d[q - 1]) / 2
        self.d, self.x = (torch.from_numpy(a).to(dev) for a in (d, x))
        gap = np.diff(x)
        self.km, self.kp = (torch.from_numpy(a).to(dev) for a in (c / (gap[1:-2] * d[2:-2]), c / (gap[2:-1] * d[2:-2])))

    def matrix(self, low, high):
        """sum of k (x_P - x_nb) along the axis; low, high: the outer value
        as a multiple of the interior one (periodic axes wrap instead)."""
        n = self.n
        m = torch.diag(self.km + self.kp) - torch.diag(self.km[1:], -1) - torch.diag(self.kp[:-1], 1)
        if self.periodic:
            m[0, n - 1] -= self.km[0]
            m[n - 1, 0] -= self.kp[-1]
        else:
            m[0, 0] -= low * self.km[0]
            m[n - 1, n - 1] -= high * self.kp[-1]
        w = torch.sqrt(self.d[2:-2])
        lam, q = torch.linalg.eigh((w[:, None] * m / w[None, :] + (w[:, None] * m / w[None, :]).T) / 2)
        return m, lam, q / w[:, None], q.T * w[None, :]


def _along(m, x, axis):
    return torch.tensordot(m, x, dims=([1], [axis])).movedim(0, axis)


class _Separable:
    """(shift + Ax + Ay + Az) x = f by the axes' eigenvectors, refined."""

    def __init__(self, axes, factors, shift):
        self.a = [ax.matrix(*f) for ax, f in zip(axes, factors)]
        lam = [a[1] for a in self.a]
        self.den = shift + lam[0][:, None, None] + lam[1][None, :, None] + lam[2][None, None, :]
        self.shift = shift
        if shift == 0.0:
            self.den.view(-1)[int(self.den.abs().argmin())] = math.inf   # the constants
            self.vol = axes[0].d[2:-2, None, None] * axes[1].d[None, 2:-2, None] * axes[2].d[None, None, 2:-2]

    def apply(self, x):
        return self.shift * x + sum(_along(a[0], x, q) for q, a in enumerate(self.a))

    def _once(self, f):
        for q, a in enumerate(self.a):
            f = _along(a[3], f, q)
        f = f / self.den
        for q, a in enumerate(self.a):
            f = _along(a[2], f, q)
        return f

    def solve(self, f, refine=3):
        x = torch.zeros_like(f)
        for _ in range(refine):
            r = f - self.apply(x)
            if self.shift == 0.0:   # the row of cell (0, 0, 0) is replaced by x = 0
                r[0, 0, 0] = 0.0
                r[0, 0, 0] = -(r * self.vol).sum() / self.vol[0, 0, 0]
            x = x + self._once(r)
            if self.shift == 0.0:
                x = x - x[0, 0, 0]
        return x


class _Exact:
    """The fractional step without a body, between walls (or a lid) and
    periodic faces, in 64 bits with its two solves done directly."""

    def __init__(self, flow):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.dt, self.re, self.dev = flow["dt"], flow["re"], dev
        self.force, self.cs = flow.get("force", (0.0, 0.0, 0.0)), flow.get("smag")
        bc = {b.split()[0]: b.split()[1:] for b in flow["bc"]}
        self.wall = [[[float(v) for v in bc[s][1:]] or [0.0] * 3 for s in pair] for pair in ("WE", "SN", "DU")]
        c = self.dt / (2 * self.re)
        self.ax = [_Axis(flow[k], bc[s][0] == "per", c, dev) for k, s in (("xf", "W"), ("yf", "S"), ("zf", "D"))]
        ratio = []   # outer velocity on a wall: (a + b)/b bc - (a/b) u, a and b half the outer and inner widths
        for a in self.ax:
            ratio.append((-float(a.d[1] / a.d[2]), -float(a.d[-2] / a.d[-3])))
        self.mom = _Separable(self.ax, ratio, 1.0)
        self.pres = _Separable(self.ax, [(1.0, 1.0)] * 3, 0.0)

    def col(self, v, axis):
        return v.reshape([-1 if a == axis else 1 for a in range(3)])

    def sh(self, x, axis, o, pad=0):
        """x at offset o along axis, over the interior (or pad layers more)."""
        ix = [slice(2 - pad, 2 - pad + a.n + 2 * pad) for a in self.ax]
        ix[axis] = slice(2 - pad + o, 2 - pad + o + self.ax[axis].n + 2 * pad)
        return x[tuple(ix)]

    def fill(self, x, comp=None):
        """Outer layers of a velocity component, or of p (comp None)."""
        for axis, a in enumerate(self.ax):
            y, d, n = x.movedim(axis, 0), a.d, a.n
            if a.periodic:
                y[1], y[0], y[n + 2], y[n + 3] = y[n + 1].clone(), y[n].clone(), y[2].clone(), y[3].clone()
            elif comp is None:
                y[1], y[0], y[n + 2], y[n + 3] = y[2].clone(), y[3].clone(), y[n + 1].clone(), y[n].clone()
            else:
                lo, hi = self.wall[axis][0][comp], self.wall[axis][1][comp]
                for o, i, e, bc in ((1, 2, (d[1] / 2, d[2] / 2), lo), (0, 3, (d[0] / 2 + d[1], d[2] + d[3] / 2), lo),
                                    (n + 2, n + 1, (d[n + 2] / 2, d[n + 1] / 2), hi),
                                    (n + 3, n, (d[n + 3] / 2 + d[n + 2], d[n + 1] + d[n] / 2), hi)):
                    y[o] = (e[0] + e[1]) / e[1] * bc - e[0] / e[1] * y[i]
        return x

    def grad(self, x, axis, pad=0):
        a = self.ax[axis]
        c = a.x[3 - pad:3 + a.n + pad] - a.x[1 - pad:1 + a.n + pad]
        return (self.sh(x, axis, 1, pad) - self.sh(x, axis, -1, pad)) / self.col(c, axis)

    def to_faces(self, x, axis):
        """x on the n + 1 faces of axis over the interior of the others; x
        padded by at least one layer along axis."""
        a = self.ax[axis]
        d = a.d[1:a.n + 3]
        return (x.narrow(axis, 0, a.n + 1) * self.col(d[1:], axis) +
                x.narrow(axis, 1, a.n + 1) * self.col(d[:-1], axis)) / self.col(d[1:] + d[:-1], axis)

    def line(self, x, axis):
        """One layer more along axis, the interior of the others."""
        return x[tuple(slice(1, a.n + 3) if q == axis else slice(2, a.n + 2) for q, a in enumerate(self.ax))]

    def face_diff(self, x, axis):
        a = self.ax[axis]
        y = self.line(x, axis)
        return (y.narrow(axis, 1, a.n + 1) - y.narrow(axis, 0, a.n + 1)) / self.col(a.x[2:a.n + 3] - a.x[1:a.n + 2], axis)

    def div(self, F):
        return sum((F[q].narrow(q, 1, a.n) - F[q].narrow(q, 0, a.n)) / self.col(a.d[2:-2], q)
                   for q, a in enumerate(self.ax))

    def conv(self, u, U):
        return [self.div([U[q] * self.to_faces(self.line(u[l], q), q) for q in range(3)]) for l in range(3)]

    def neighbours(self, x):
        return sum(self.col(a.km, q) * (self.sh(x, q, -1) - self.sh(x, q, 0)) +
                   self.col(a.kp, q) * (self.sh(x, q, 1) - self.sh(x, q, 0)) for q, a in enumerate(self.ax))

    def pad(self, x, comp):
        return self.fill(torch.nn.functional.pad(x, (2,) * 6), comp)

    def stress(self, u):
        """Divergence of the Smagorinsky stress, zero outside the grid."""
        g = [[self.grad(u[l], q) for q in range(3)] for l in range(3)]
        s = [[(g[l][q] + g[q][l]) / 2 for q in range(3)] for l in range(3)]
        mag = torch.sqrt(sum(2 * s[l][q] ** 2 for l in range(3) for q in range(3)))
        d = [self.col(a.d[2:-2], q) for q, a in enumerate(self.ax)]
        length = torch.clamp(self.cs * 2 * (d[0] * d[1] * d[2]) ** (1 / 3), max=0.41 * 0.5)
        return [sum(self.grad(torch.nn.functional.pad(-2 * length ** 2 * mag * s[l][q], (2,) * 6), q)
                    for q in range(3)) for l in range(3)]

    def iterate(self, state, steps):
        dt = self.dt
        u = [self.fill(torch.as_tensor(np.array(x), device=self.dev), l) for l, x in enumerate(state[:3])]
        p = self.fill(torch.as_tensor(np.array(state[3]), device=self.dev))
        U = [self.to_faces(self.line(u[q], q), q) for q in range(3)]
        last = self.conv(u, U)
        for _ in range(steps):
            now = self.conv(u, U)
            tau = self.stress(u) if self.cs is not None else (0.0, 0.0, 0.0)
            us = []
            for l in range(3):
                b = (-dt / 2 * (3 * now[l] - last[l]) - dt * self.grad(p, l) + self.sh(u[l], 0, 0) +
                     self.neighbours(u[l]) + dt * self.force[l] - dt * tau[l])
                for axis, a in enumerate(self.ax):   # the walls' share of the rows beside them
                    if a.periodic:
                        continue
                    lo, hi = self.wall[axis][0][l], self.wall[axis][1][l]
                    b.select(axis, 0).add_(float(a.km[0] * (a.d[1] + a.d[2]) / a.d[2]) * lo)
                    b.select(axis, a.n - 1).add_(float(a.kp[-1] * (a.d[-2] + a.d[-3]) / a.d[-3]) * hi)
                us.append(self.pad(self.mom.solve(b), l))
            Us = []
            for q in range(3):
                t = self.sh(us[q], 0, 0, 1) + dt * self.grad(p, q, 1)
                t = t[tuple(slice(None) if r == q else slice(1, -1) for r in range(3))]
                Us.append(self.to_faces(t, q) - dt * self.face_diff(p, q))
            pp = self.pad(self.pres.solve(-self.div(Us) / (2 * self.re)), None)
            U = [Us[q] - dt * self.face_diff(pp, q) for q in range(3)]
            u = [self.pad(self.sh(us[l], 0, 0) - dt * self.grad(pp, l), l) for l in range(3)]
            p = self.fill(p + pp)
            last = now
        return u + [p]


def exact(case, seed):
    """The same steps in 64 bits with direct solves.  With a body the level
    set of its STL, the ghost stencils and their ordered in-place updates
    would come first and the solves lose their direct form: in plain torch
    far over 20 seconds, so None."""
    if case["flow"] not in ("cavity", "channel"):
        return None
    flow = _flow(case)
    return [_Exact(flow).iterate(_initial(flow, seed), case["steps"])]
