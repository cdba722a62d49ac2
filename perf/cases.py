"""Timed cases of the PU-RBF interpolation and advection path, through the public Python API.

A case is one pass of what a user's program repeats:

  job         advected particles for a resident dataset (what the serving loop runs per job): new
              particles in, the velocity at them, a few steps of an RK scheme, their positions out.
  resident    one step of a long run: the particles stay on the device, the step is advanced and the
              positions are written out.
  interp      one snapshot: new field values for the data points, the patch set-ups (or the re-solve
              with kept factors) and the interpolated fields at a new set of points.
  step        one step of AdvectionInterpolation over a new particle set: data in, interpolation,
              fields out, advection to the next time, positions out.
  analytical  one step in a device-side analytical velocity field.

Sizes: `nlat` lattice points per axis (or `nd` points of the Gaussian mixture), `npu` PU nodes per
axis (overlap 1.5 spacings), `np` particles, `steps` intervals of `dt` with the RK scheme `scheme`
(0 RK1, 1 RK2, 2 RK4, 3 Dormand-Prince), `kernel` 2 Wendland C2 or 6 Gaussian with eps = `gauss`
lattice spacings^-1, `solve` 2 set-up on every snapshot (the Python default) or 1 factors kept,
`fp32` the FP32 evaluation.  The path takes and returns host arrays, so inputs and outputs are host
arrays; interpolated fields of the FP32 evaluation, which carry FP32 precision, are kept as float32.
"""
import math

import numpy as np
import torch

import lagrbf_gb300 as L
from lagrbf_gb300 import workloads as W

BASE = dict(kind="job", dim=3, data="lattice", nd=0, nlat=0, npu=0, np=0, kernel=2, gauss=0.0, nfields=3, fp32=True,
            solve=2, scheme=2, steps=1, dt=5e-4)


def _case(name=None, **kw):
    c = dict(BASE, **kw)
    if c["data"] == "lattice":
        c["nd"] = c["nlat"] ** c["dim"]
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the 2D plain configuration, one outer step of the drop-in call sequence with its defaults
        _case("step 2D gauss fp64", kind="step", dim=2, nlat=64, npu=8, np=10_000, kernel=6, gauss=3.0, nfields=2,
              fp32=False, dt=1e-3),
        # the smallest job of the serving mix: latency and launches
        _case("job 1K rk2", nlat=22, npu=6, np=1_000, scheme=1, steps=4),
        # its median job: 100K particles on a dataset of 150K points
        _case("job 100K rk4", nlat=53, npu=14, np=100_000, scheme=2, steps=2),
        # a large job with Dormand-Prince on a 1M-point dataset
        _case("job 2M dp45", nlat=100, npu=25, np=2_000_000, scheme=3, steps=1),
        # the headline configuration: 2.1M points, 16.8M particles, RK4 with FP32 evaluation
        _case("resident 16.8M rk4", kind="resident", nlat=128, npu=32, np=16_777_216),
        # plain FP64 advection of a moderate set
        _case("job fp64 200K rk4", nlat=64, npu=16, np=200_000, fp32=False),
        # one-shot FP64 interpolation with its patch set-ups: a scalar and a vector field (4 components)
        _case("interp 3D 4 fields fp64", kind="interp", nlat=48, npu=12, np=50_000, nfields=4, fp32=False),
        # a scalar on a large 2D dataset, ragged sizes
        _case("interp 2D scalar fp64", kind="interp", dim=2, nlat=301, npu=37, np=300_007, nfields=1, fp32=False),
        # time-dependent values on fixed points: re-solve with kept factors, FP32 evaluation
        _case("interp re-solve fp32", kind="interp", nlat=64, npu=16, np=1_000_000, solve=1),
        # the precision-stress configuration: Gaussian kernel, few points per cell
        _case("job gauss 4M rk4", nlat=80, npu=32, np=4_000_000, kernel=6, gauss=1.0),
        # uneven data: Gaussian mixture, patches from a few points to many hundreds
        _case("job mixture 1M rk4", data="mixture", nd=250_000, npu=100, np=1_000_000),
        # a device-side analytical field: stages and particle bookkeeping without the evaluation
        _case("analytical 2D 4M", kind="analytical", dim=2, npu=64, np=4_000_000, nfields=2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["job", "job", "job", "interp", "interp", "step", "analytical"])
    if kind == "analytical":
        return _case(kind=kind, dim=2, npu=rng.randrange(3, 129), nfields=2, np=_log_int(rng, 1e3, 4e6),
                     scheme=rng.choice([0, 1, 2, 3]))
    if kind == "job":
        fp32 = rng.random() < 0.75
        nlat = _log_int(rng, 16, 100)
        per_cell = rng.uniform(20.0, 90.0)
        npu = max(3, int(round((nlat ** 3 / per_cell) ** (1 / 3))) + 1)
        gauss = rng.random() < 0.25
        return _case(kind=kind, nlat=nlat, npu=npu, np=_log_int(rng, 1e3, 4e6 if fp32 else 3e5), fp32=fp32,
                     kernel=6 if gauss else 2, gauss=1.0 if gauss else 0.0, scheme=rng.choice([0, 1, 2, 2, 3]),
                     steps=rng.randrange(1, 4))
    dim = rng.choice([2, 3])
    per_cell = rng.uniform(20.0, 90.0)
    nlat = _log_int(rng, 20, 400) if dim == 2 else _log_int(rng, 12, 60)
    npu = max(3, int(round((nlat ** dim / per_cell) ** (1 / dim))) + 1)
    fp32 = rng.random() < 0.5
    solve = rng.choice([1, 2])
    if kind == "interp":
        return _case(kind=kind, dim=dim, nlat=nlat, npu=npu, np=_log_int(rng, 1e3, 2e6 if fp32 else 2e5),
                     nfields=rng.choice([1, dim, dim, dim + 1]), fp32=fp32, solve=solve)
    return _case(kind=kind, dim=dim, nlat=min(nlat, 200 if dim == 2 else 40),
                 npu=npu if nlat <= (200 if dim == 2 else 40) else max(3, npu // 2), np=_log_int(rng, 1e3, 1e5),
                 nfields=dim, fp32=fp32, solve=solve, scheme=rng.choice([1, 2, 3]), dt=1e-3)


# ------------------------------------------------------------------------------------- inputs
def _inputs(c, seed):
    """Data points and values, and particles: seeded, host arrays."""
    rng = np.random.default_rng(seed)
    dim = c["dim"]
    xd = fd = None
    if c["kind"] != "analytical":
        if c["data"] == "mixture":
            clusters = W.mixture_clusters(3, np.random.default_rng(5))
            xd = W.mixture_points(c["nd"], 3, rng, clusters=clusters)
        else:
            xd = W.jittered_lattice(c["nlat"], dim, rng)
        vel = W.abc_flow(xd) if dim == 3 else W.cellular_flow(xd)
        extra = np.sin(2.0 * np.pi * (xd @ rng.integers(1, 4, dim)) + rng.uniform(0.0, 2.0 * np.pi))[:, None]
        fd = np.ascontiguousarray(extra if c["nfields"] == 1 else np.concatenate([vel, extra], 1)[:, :c["nfields"]])
    if c["data"] == "mixture":
        xp = W.mixture_points(c["np"], 3, rng, clusters=clusters)
    else:
        xp = rng.random((c["np"], dim))
    return xd, fd, xp


def _eps(c):
    """Support radius of the PU weights (1.5 node spacings), 1/radius and the RBF shape parameter."""
    rad = W.pu_overlap(c["npu"]) / c["npu"]
    eps_w = 1.0 / rad
    return rad, eps_w, (c["gauss"] * c["nlat"] if c["kernel"] == 6 else eps_w)


class State:
    pass


def prepare(case, seed):
    c = case
    s = State()
    s.case, s.t = c, 0.0
    xd, fd, s.xp = _inputs(c, seed)
    _, eps_w, eps_r = _eps(c)
    kind, n, dim = c["kind"], c["np"], c["dim"]
    opts = dict(dim=dim, npartitions=[c["npu"]] * dim, overlap=W.pu_overlap(c["npu"]), shape_factor=eps_r / eps_w,
                kernel=c["kernel"], nfields=c["nfields"], solve_method=c["solve"],
                eval_precision="fp32" if c["fp32"] else "fp64", advection=kind != "interp",
                advection_scheme=c["scheme"], advection_cfl=0.3, dt=c["dt"])
    # resident datasets are set up whole, as the serving loop keeps them
    s.ctx = L.LagRBFCtx({"setup_all_patches": kind in ("job", "resident")}, **opts)
    s.pid = np.arange(1, n + 1, dtype=np.int64)
    s.x = np.full((n, dim), 0.0)                  # caller-allocated output rows, touched
    s.f = np.full((n, c["nfields"]), 0.0)
    s.f32 = torch.zeros((n, c["nfields"]), dtype=torch.float32)
    s.xd, s.fd = xd, fd
    if kind in ("job", "resident"):
        s.ctx.fill_data(xd, fd)
        s.ctx.fill_points(s.xp, pidx=s.pid)
        s.ctx.interpolate_c()                     # sets every patch up
    elif kind == "interp":
        if c["solve"] == 1:                       # the factors a user keeps between snapshots
            s.ctx.fill_data(xd, fd)
            s.ctx.fill_points(s.xp, pidx=s.pid)
            s.ctx.interpolate_c()
    elif kind == "step":
        if c["solve"] == 1:
            s.ctx.fill_data(xd, fd)
            s.ctx.fill_points(s.xp, pidx=s.pid)
            s.ctx.interpolate_c()
            s.ctx.reset_coefficients()
    else:
        s.ctx.set_velocity_field(s.ctx.VFIELD_CELLULAR, [1.0, 1.0])
        s.ctx.fill_points(s.xp, pidx=s.pid)
    return s


def _fields(s):
    """Interpolated fields by pid; single precision is kept where the evaluation is."""
    s.ctx.output(fvals=s.f)
    if not s.case["fp32"]:
        return s.f
    return s.f32.copy_(torch.from_numpy(s.f))


def run(s):
    c, ctx = s.case, s.ctx
    kind, dt = c["kind"], c["dt"]
    if kind == "job":
        ctx.fill_points(s.xp, pidx=s.pid)
        ctx.interpolate_c()
        for k in range(c["steps"]):
            ctx.advect_resident(k * dt, (k + 1) * dt)
        ctx.output(coords=s.x)
        return {"x": s.x}
    if kind == "resident":
        ctx.advect_resident(s.t, s.t + dt)
        s.t += dt
        ctx.output(coords=s.x)
        return {"x": s.x}
    if kind == "interp":
        ctx.reset_coefficients()
        ctx.fill_data(s.xd, s.fd)
        ctx.fill_points(s.xp, pidx=s.pid)
        ctx.interpolate_c()
        return {"f": _fields(s)}
    if kind == "step":
        ctx.fill_points(s.xp, pidx=s.pid)
        ctx.fill_data(s.xd, s.fd)
        ctx.interpolate_c()
        f = _fields(s)
        ctx.advect_interpolate_c(0.0, dt)
        ctx.output(coords=s.x)
        return {"f": f, "x": s.x}
    ctx.advect_analytical_c(s.t, s.t + dt)
    s.t += dt
    ctx.output(coords=s.x, fvals=s.f, fieldname="velocity")
    return {"x": s.x, "v": s.f}


# ------------------------------------------------------------------------------------- floors
EVALS = {0: 1, 1: 2, 2: 4, 3: 8}  # evaluations of a step, the fields at its end among them


def _evals(c):
    e = EVALS[c["scheme"]] * c["steps"]
    return {"job": 1 + e, "resident": e, "interp": 1, "step": 1 + e, "analytical": 0}[c["kind"]]


def _patch(c):
    """Points per cell and in an inner patch, cells and nodes."""
    cells = (c["npu"] - 1) ** c["dim"]
    per = c["nd"] / cells
    return per, per * 2 ** c["dim"], cells, c["npu"] ** c["dim"]


def work(case):
    """Bytes: inputs read and outputs written once.  Flops: of each (particle, data point) pair inside
    the kernel's support the distance and kernel (18) and 2 per coefficient (a point lies in
    (4/3)^dim patches of the particle's cell on average); m^3/3 + 2 F m^2 per patch set up (the solve
    alone with kept factors); the particle updates of the stages."""
    c = case
    dim, n, F, kind = c["dim"], c["np"], c["nfields"], c["kind"]
    rows = {"job": 2 * dim, "resident": 2 * dim, "interp": dim + F, "step": 2 * dim + F, "analytical": 3 * dim}[kind]
    by = 8.0 * n * rows
    if kind == "analytical":
        return {"bytes": by, "flops": 40.0 * n * EVALS[c["scheme"]]}
    per, m, cells, nodes = _patch(c)
    if c["data"] == "mixture":  # points per cell as a particle of the same mixture meets them
        rng, clusters = np.random.default_rng(0), W.mixture_clusters(3, np.random.default_rng(5))
        a, b = (_PU.flat([(W.mixture_points(100_000, 3, rng, clusters=clusters)[:, d] * (c["npu"] - 1)).astype(np.int64)
                          .clip(0, c["npu"] - 2) for d in range(3)], c["npu"] - 1) for _ in range(2))
        per = c["nd"] * float(np.dot(np.bincount(a, minlength=cells) / a.size, np.bincount(b, minlength=cells) / b.size))
    ball = {2: math.pi, 3: 4.0 / 3.0 * math.pi}[dim] * 1.5 ** dim
    pairs = n * per * (3.0 ** dim if c["kernel"] == 6 else min(ball, 3.0 ** dim))
    Fe = dim if kind in ("job", "resident") else F
    fl = pairs * (18.0 + 2.0 * Fe * (4.0 / 3.0) ** dim) * _evals(c)
    if kind in ("interp", "step"):
        by += 8.0 * c["nd"] * (dim + F)
        inner = (1.0 - 1.0 / c["npu"]) ** dim  # share of a full patch on average (boundary nodes hold fewer cells)
        fl += nodes * ((m * inner) ** 3 / 3.0 if c["solve"] == 2 else 0.0) + nodes * 2.0 * F * (m * inner) ** 2
    return {"bytes": by, "flops": fl}


# ------------------------------------------------------------------------- 64-bit restatement
class _PU:
    """The PU-RBF interpolant in plain float64 torch: per-patch collocation, Cholesky, weighted sum."""

    def __init__(self, c, xd, fd, dev):
        self.c, self.dev, self.dim, self.n = c, dev, c["dim"], c["npu"]
        self.rad, self.eps_w, self.eps_r = _eps(c)
        self.h = 1.0 / (self.n - 1)
        xd, fd = torch.from_numpy(xd).to(dev), torch.from_numpy(fd).to(dev)
        dim, n, nc = self.dim, self.n, self.n - 1
        cell = self.flat(self.cells(xd), nc)
        order = torch.argsort(cell, stable=True)
        self.xs, self.fs = xd[order], fd[order]
        count = torch.bincount(cell, minlength=nc ** dim)
        start = torch.cumsum(count, 0) - count
        # index rows of every patch (adjacent cells in ascending order), padded with -1
        node = torch.arange(n ** dim, device=dev)
        ijk = [(node // n ** d) % n for d in range(dim)]
        first, num = [], []
        for s in range(2 ** dim):
            cc = [ijk[d] - 1 + ((s >> d) & 1) for d in range(dim)]
            ok = torch.ones_like(node, dtype=torch.bool)
            for v in cc:
                ok &= (v >= 0) & (v < nc)
            f = torch.where(ok, self.flat([v.clamp(0, nc - 1) for v in cc], nc), 0)
            first.append(start[f])
            num.append(torch.where(ok, count[f], 0))
        self.m = torch.stack(num).sum(0)
        self.mmax = int(self.m.max())
        q = torch.arange(self.mmax, device=dev)[None, :]
        self.idx = torch.full((n ** dim, self.mmax), -1, dtype=torch.int64, device=dev)
        off = torch.zeros_like(node)
        for f, k in zip(first, num):
            inside = (q >= off[:, None]) & (q < (off + k)[:, None])
            self.idx = torch.where(inside, f[:, None] + q - off[:, None], self.idx)
            off = off + k
        self.X = torch.zeros((n ** dim, self.mmax, fd.shape[1]), dtype=torch.float64, device=dev)
        step = max(1, int(1.5e8 / self.mmax ** 2))
        for a in range(0, n ** dim, step):
            ix = self.idx[a:a + step]
            live = ix >= 0
            p = self.xs[ix.clamp(min=0)]
            d2 = torch.zeros((ix.shape[0], self.mmax, self.mmax), dtype=torch.float64, device=dev)
            for d in range(dim):
                d2 += (p[:, :, None, d] - p[:, None, :, d]) ** 2
            A = self.phi(d2)
            A = torch.where(live[:, :, None] & live[:, None, :], A, 0.0)
            A += torch.diag_embed((~live).to(torch.float64))
            rhs = torch.where(live[:, :, None], self.fs[ix.clamp(min=0)], 0.0)
            self.X[a:a + step] = torch.cholesky_solve(rhs, torch.linalg.cholesky(A))

    def cells(self, x):
        t = torch.floor(x / self.h).to(torch.int64).clamp(0, self.n - 2)
        return [t[:, d] for d in range(self.dim)]

    @staticmethod
    def flat(ijk, n):
        return sum(v * n ** d for d, v in enumerate(ijk))

    def phi(self, d2):
        if self.c["kernel"] == 6:
            return torch.exp(-(self.eps_r ** 2) * d2)
        return self.c2(d2, self.eps_r)

    @staticmethod
    def c2(d2, eps):
        u = (1.0 - eps * torch.sqrt(d2)).clamp(min=0.0)
        return u ** 4 * (5.0 - 4.0 * u)

    def __call__(self, x, nf):
        out = torch.empty((x.shape[0], nf), dtype=torch.float64, device=self.dev)
        step = max(1, int(6e7 / self.mmax))
        for a in range(0, x.shape[0], step):
            out[a:a + step] = self.part(x[a:a + step], nf)
        return out

    def part(self, x, nf):
        dim, n = self.dim, self.n
        ci = self.cells(x)
        den = torch.zeros(x.shape[0], dtype=torch.float64, device=self.dev)
        for o in range(6 ** dim):
            d2, ok = torch.zeros_like(den), torch.ones_like(den, dtype=torch.bool)
            for d in range(dim):
                i = ci[d] + (o // 6 ** d) % 6 - 2
                ok &= (i >= 0) & (i < n)
                d2 += (x[:, d] - self.h * i.double()) ** 2
            den += torch.where(ok, self.c2(d2, self.eps_w), 0.0)
        val = torch.zeros((x.shape[0], nf), dtype=torch.float64, device=self.dev)
        for k in range(2 ** dim):
            ijk = [ci[d] + ((k >> d) & 1) for d in range(dim)]
            w2 = sum((x[:, d] - self.h * ijk[d].double()) ** 2 for d in range(dim))
            w = self.c2(w2, self.eps_w) / den
            node = self.flat(ijk, n)
            ix = self.idx[node]
            p = self.xs[ix.clamp(min=0)]
            d2 = sum((x[:, None, d] - p[:, :, d]) ** 2 for d in range(dim))
            ph = torch.where(ix >= 0, self.phi(d2), 0.0)
            val += w[:, None] * torch.bmm(ph[:, None, :], self.X[node][:, :, :nf])[:, 0]
        return val


_DP_A = [[1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9],
         [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
         [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656],
         [35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]]


def _advance(c, x, vel, cfl_radius, intervals, alive):
    """x after the intervals (t, t_next) of the scheme; particles that leave [0, 1]^dim are removed."""
    v = vel(x)

    def keep(y):
        alive.logical_and_(((y >= 0) & (y <= 1)).all(1))
        return torch.where(alive[:, None], y, 0.5)

    for t, t_next in intervals:
        while t < t_next:
            dt = 0.3 * cfl_radius / (float(v[alive].norm(dim=1).max()) + 1e-16)
            if c["scheme"] == 3:
                dt = min(dt, t_next - t)  # the error control allows the whole interval
            if t + dt > t_next:
                dt = t_next - t
            if c["scheme"] == 0:
                x = keep(x + dt * v)
            elif c["scheme"] == 1:
                x = keep(x + dt * vel(keep(x + 0.5 * dt * v)))
            elif c["scheme"] == 2:
                k = [v]
                for f in (0.5, 0.5, 1.0):
                    k.append(vel(keep(x + f * dt * k[-1])))
                x = keep(x + dt / 6.0 * (k[0] + 2.0 * k[1] + 2.0 * k[2] + k[3]))
            else:
                k = [v]
                for row in _DP_A:
                    y = keep(x + dt * sum(a * b for a, b in zip(row, k)))
                    k.append(vel(y))
                x = y
            v = vel(x)
            t = t + dt
    return x, v


def exact(case, seed):
    c = case
    dim, kind, n = c["dim"], c["kind"], c["np"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    rad = _eps(c)[0]
    if kind == "analytical":
        x = torch.from_numpy(_inputs(c, seed)[2]).to(dev)
        alive = torch.ones(n, dtype=torch.bool, device=dev)

        def cellular(y):
            px, py = math.pi * y[:, 0], math.pi * y[:, 1]
            return torch.stack([torch.sin(px) * torch.cos(py), -torch.cos(px) * torch.sin(py)], 1)

        # the velocity of the swarm starts from the field at the particles
        x, v = _advance(c, x, cellular, rad, [(0.0, c["dt"])], alive)
        return {"x": torch.where(alive[:, None], x, 0.0), "v": torch.where(alive[:, None], v, 0.0)}
    per, m, cells, nodes = _patch(c)
    if c["data"] == "mixture" or n * m * 2 ** dim * _evals(c) > 3e11 or nodes * m ** 3 / 3 > 6e11:
        return None
    xd, fd, xp = _inputs(c, seed)
    pu = _PU(c, xd, fd, dev)
    x = torch.from_numpy(xp).to(dev)
    if kind == "interp":
        return {"f": pu(x, c["nfields"])}
    alive = torch.ones(n, dtype=torch.bool, device=dev)
    dt = c["dt"]
    steps = 1 if kind in ("step", "resident") else c["steps"]
    y, _ = _advance(c, x, lambda z: pu(z, dim), rad, [(k * dt, (k + 1) * dt) for k in range(steps)], alive)
    y = torch.where(alive[:, None], y, 0.0)
    return {"f": pu(x, c["nfields"]), "x": y} if kind == "step" else {"x": y}
