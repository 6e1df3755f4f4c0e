"""The work a user of this engine has it do, as timed cases.

Every case goes through the package's public calls on seeded synthetic
structures of the kinds the engine is used for: SOI guides and grating
couplers in 2D, pixel design regions, pillar metasurfaces and strip guides in
3D, batches and served streams of such jobs, and the frequency-domain solver
with its adjoint.

  listed()            the cases
  draw(rng)           one more case of the same ranges
  prepare(case, seed) a program's inputs and handles before the call
  run(state)          one pass
  work(case)          bytes and operations a pass cannot do without
  exact(case, seed)   the results in 64 bits, by plain torch

All runs have a fixed number of steps (shutoff 0), so a pass is the same work
for every seed.
"""
from __future__ import annotations

import math
import warnings

import numpy as np
import torch

from opticrcwafdtd_b200 import (Context, Job, NotConvergedWarning, Server, epsComponents2D, epsComponents3D, epsFromBoxes,
                                fdfd2D, fdtd2D, fdtd2D_batch, fdtd3D, workloads)

warnings.simplefilter("ignore", NotConvergedWarning)   # fixed step counts end at maxTime

N_SI, N_OX = 3.476, 1.444


# ------------------------------------------------------------------- cases --
def listed() -> list[dict]:
    return [
        # the smallest call: a plane wave on a slab, periodic in z (a validation run, a sweep's cheap point)
        dict(name="slab_te_fp64", kind="slab", nx=601, nz=4, steps=1500, precision="double", n_lambda=7),
        # one SOI grating coupler, the reference's default design run, double precision
        dict(name="coupler_te_fp64", kind="coupler", nx=800, nz=300, steps=4000, precision="double", n_lambda=51),
        # a pixel design region, the largest 2D run, advanced as a device-resident job
        dict(name="pixel_tm_fp32", kind="pixel", nx=4000, nz=1500, steps=4000, precision="single", n_lambda=101),
        # a pixel region of ragged size in double precision, whole call
        dict(name="pixel_tm_fp64_odd", kind="pixel_call", nx=1611, nz=707, steps=1500, precision="double", n_lambda=11),
        # a design sweep: many uneven couplers in one call
        dict(name="coupler_batch_fp32", kind="batch", n=32, steps=3000, precision="single", n_lambda=51),
        # a served stream: mixed 2D couplers and 3D unit cells of uneven size, submitted at once
        dict(name="serve_mixed_fp32", kind="serve", n=8, steps=1000, precision="single", n_lambda=11),
        # a pillar metasurface, the largest 3D run, advanced as a device-resident job
        dict(name="pillar_fp32", kind="pillar", nx=600, ny=600, nz=300, steps=240, precision="single", n_lambda=1),
        # a smaller lattice, double precision, whole call from host arrays
        dict(name="pillar_fp64_call", kind="pillar_call", nx=200, ny=160, nz=141, steps=400, precision="double", n_lambda=3),
        # one metalens unit cell (periodic x and y): the point of a phase library
        dict(name="unit_cell_fp32", kind="cell", nx=22, ny=22, nz=171, steps=2000, precision="single", n_lambda=3),
        # a strip guide with absorbing layers on all six sides, odd sizes
        dict(name="strip_fp32", kind="strip", nx=201, ny=93, nz=77, steps=1000, precision="single", n_lambda=5),
        # a new frequency-domain problem: factor the operator and solve once
        dict(name="fdfd_factor", kind="fdfd", nx=501, nz=221),
        # an inverse-design step on kept factors: another current, then the adjoint
        dict(name="fdfd_solve_adjoint", kind="fdfd_solves", nx=501, nz=221),
    ]


def _log(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["slab", "coupler", "coupler", "pixel", "pixel_call", "batch", "serve", "pillar", "pillar_call",
                       "cell", "strip", "fdfd", "fdfd", "fdfd_solves"])
    prec = rng.choice(["single", "single", "double"])
    if kind == "slab":
        return dict(kind=kind, nx=_log(rng, 300, 1500), nz=rng.randint(3, 9), steps=rng.randint(600, 2500), precision=prec,
                    n_lambda=rng.randint(3, 13))
    if kind == "coupler":
        return dict(kind=kind, nx=_log(rng, 420, 2000), nz=rng.randint(220, 560), steps=rng.randint(1000, 4000),
                    precision=prec, n_lambda=rng.randint(5, 51))
    if kind in ("pixel", "pixel_call"):
        big = 1 if prec == "single" else 0.7
        return dict(kind=kind, nx=_log(rng, 1400, 3900 * big), nz=_log(rng, 400, 1400 * big), steps=rng.randint(600, 2000),
                    precision=prec, n_lambda=rng.randint(5, 101))
    if kind == "batch":
        return dict(kind=kind, n=rng.randint(6, 32), steps=rng.randint(800, 2500), precision=prec, n_lambda=rng.randint(5, 51))
    if kind == "serve":
        return dict(kind=kind, n=rng.randint(4, 10), steps=rng.randint(500, 1200), precision="single", n_lambda=11)
    if kind == "pillar":
        return dict(kind=kind, nx=20 * rng.randint(8, 26), ny=20 * rng.randint(8, 26), nz=rng.randint(130, 290),
                    steps=rng.randint(200, 240), precision=prec, n_lambda=rng.randint(1, 3))
    if kind == "pillar_call":
        return dict(kind=kind, nx=20 * rng.randint(5, 12), ny=20 * rng.randint(5, 12), nz=rng.randint(125, 190),
                    steps=rng.randint(220, 400), precision=prec, n_lambda=rng.randint(1, 5))
    if kind == "cell":
        return dict(kind=kind, nx=rng.randint(14, 40), ny=rng.randint(14, 40), nz=rng.randint(110, 260),
                    steps=rng.randint(800, 2000), precision=prec, n_lambda=rng.randint(1, 7))
    if kind == "strip":
        return dict(kind=kind, nx=rng.randint(90, 320), ny=rng.randint(61, 121), nz=rng.randint(61, 101),
                    steps=rng.randint(400, 1000), precision=prec, n_lambda=rng.randint(1, 5))
    # the shorter axis of the frequency-domain grids up to the solver's limit of 384
    nx, nz = _log(rng, 150, 600), rng.randint(90, 250)
    if rng.random() < 0.15:
        nx, nz = rng.randint(257, 300), rng.randint(257, 300)
    if rng.random() < 0.3:
        nx, nz = nz, nx
    return dict(kind=kind, nx=nx, nz=nz)


# ------------------------------------------------------------------ inputs --
def _slab_sim(c, seed):
    """A plane wave through a slab, periodic in z (10 nm grid)."""
    r = np.random.default_rng(seed)
    dx, nx, nz = 0.01, c["nx"], c["nz"]
    x, z = np.arange(nx) * dx, np.arange(nz) * dx
    x1 = (0.45 + 0.1 * r.random()) * nx * dx
    eps = epsFromBoxes(x, z, 1.0, [x1, x1 + r.uniform(0.2, 0.6), -np.inf, np.inf, r.uniform(1.4, 3.5)])
    S = 0.99 / math.sqrt(2) * dx
    return dict(pol="TE", x=x, z=z, eps=eps, npml=[20, 0], periodicZ=True, lambdas=np.linspace(1.2, 1.8, c["n_lambda"]),
                monitors=[61, nx - 60], maxTime=c["steps"] * S, shutoff=0.0, precision=c["precision"],
                source=dict(ix=101, profile=np.ones(nz), neff=1.0, lambda0=1.5, bw=0.3))


def _coupler_sim(c, r):
    """An SOI grating coupler with its own period, fill and etch (20 nm grid)."""
    dx, nx, nz = 0.02, c["nx"], c["nz"]
    period, ff, etch = r.uniform(0.56, 0.70), r.uniform(0.3, 0.7), r.uniform(0.05, 0.12)
    x = np.arange(nx) * dx
    z = np.arange(nz) * dx - 0.4 * nz * dx + dx / 2
    box = min(2.0, 0.35 * nz * dx)
    boxes = workloads.grating_coupler_geometry(period, ff, etch, n_per=max(4, int((nx * dx - 4.0) / period)), x_start=2.5,
                                               n_clad=N_OX, box=box)
    eps = epsComponents2D(x, z, N_OX, boxes)["y"]
    ix = 51
    neff, prof = workloads.core_mode(z, np.sqrt(eps[ix - 1, :]), 1.55, substrate_top=-box)
    S = 0.99 / math.sqrt(2) * dx
    kup, kdn = int(np.argmin(np.abs(z - 1.22))) + 1, int(np.argmin(np.abs(z + 1.0))) + 1
    return dict(pol="TE", x=x, z=z, eps=eps, npml=[20, 20], lambdas=np.linspace(1.5, 1.6, c["n_lambda"]),
                monitors=[ix - 25, ix + 10, nx - 30], monitorsZ=[kup, kdn], maxTime=c["steps"] * S, shutoff=0.0,
                precision=c["precision"], source=dict(ix=ix, profile=prof, neff=neff, lambda0=1.55, bw=0.05 / 1.55))


def _pixel_sim(c, seed):
    sim = workloads.pixel_region_sim(seed=seed, steps=c["steps"], precision=c["precision"], nx=c["nx"], nz=c["nz"],
                                     n_lambda=c["n_lambda"])
    # a short pulse, so that a bounded run has it in the design region, at an amplitude of the seed's own
    sim["source"].update(bw=0.3, profile=sim["source"]["profile"] * np.random.default_rng(seed).uniform(0.5, 1.5))
    mid = round(0.5 * c["nz"])
    sim["monitorsZ"] = [mid + c["nz"] // 6, mid - c["nz"] // 6]
    return sim


def _batch_sims(c, seed):
    r = np.random.default_rng(seed)
    size = np.random.default_rng(1000 + c["n"])   # the sizes are the case's, the structures the seed's
    return [_coupler_sim(dict(c, nx=int(size.integers(600, 1201)), nz=int(size.integers(250, 351))), r) for _ in range(c["n"])]


def _pillar_sim(c, seed, ctx):
    sim = workloads.pillar_lattice_sim(nx=c["nx"], ny=c["ny"], nz=c["nz"], seed=seed, steps=c["steps"],
                                       precision=c["precision"], n_lambda=c["n_lambda"], device=ctx)
    sim["source"]["bw"] = 0.6   # a short pulse: a bounded run has it past the pillars
    return sim


def _cell_sim(c, seed, ctx):
    """One pillar on a substrate, periodic in x and y, plane wave toward +z."""
    r = np.random.default_rng(seed)
    d, nx, ny, nz = 0.02, c["nx"], c["ny"], c["nz"]
    x, y, z = (np.arange(nx) + 0.5) * d, (np.arange(ny) + 0.5) * d, np.arange(nz) * d
    zs = 0.3 * nz * d
    P = nx * d
    wx, wy = r.uniform(0.3, 0.8) * P, r.uniform(0.3, 0.8) * ny * d
    shapes = [["box", [-np.inf, np.inf, -np.inf, np.inf, -np.inf, zs, 1.46]],
              ["box", [P / 2 - wx / 2, P / 2 + wx / 2, (ny * d - wy) / 2, (ny * d + wy) / 2, zs, zs + 0.6, 2.4]]]
    e = epsComponents3D(x, y, z, 1.0, shapes)
    S = 0.99 / math.sqrt(3) * d
    i0 = int(zs / d) - 8
    src = dict(axis=3, index=i0, Ea=1.0, Eb=0.0, Ha=0.0, Hb=1.46, neff=1.46, lambda0=0.532, bw=0.1)
    mons = [dict(axis=3, index=i0 - 4), dict(axis=3, index=nz - 16)]
    return dict(x=x, y=y, z=z, eps=e, npml=[0, 0, 12], periodic=[True, True, False], source=src, monitors=mons,
                lambdas=np.linspace(0.51, 0.55, c["n_lambda"]), maxTime=c["steps"] * S, shutoff=0.0, precision=c["precision"])


def _strip_sim(c, seed):
    """A strip guide along x with a scatterer on it, CPML on all sides."""
    r = np.random.default_rng(seed)
    d, nx, ny, nz = 0.04, c["nx"], c["ny"], c["nz"]
    x, y, z = np.arange(nx) * d, (np.arange(ny) - (ny - 1) / 2) * d, (np.arange(nz) - (nz - 1) / 2) * d
    w, h = r.uniform(0.2, 0.35), 0.11
    xs = r.uniform(0.45, 0.6) * nx * d
    shapes = [["box", [-np.inf, np.inf, -w, w, -h, h, N_SI]],
              ["box", [xs, xs + r.uniform(0.1, 0.4), -w, w, h, h + 0.2, r.uniform(1.8, 3.4)]]]
    e = epsComponents3D(x, y, z, N_OX, shapes)
    f = np.exp(-(y[:, None] / (1.4 * w)) ** 2 - (z[None, :] / 0.22) ** 2)
    S = 0.99 / math.sqrt(3) * d
    src = dict(axis=1, index=16, Ea=f, Eb=0.05 * f, Ha=-0.1 * f, Hb=2.3 * f, neff=2.3, lambda0=1.55, bw=0.1)
    mons = [dict(axis=1, index=12), dict(axis=1, index=26), dict(axis=1, index=nx - 14), dict(axis=3, index=nz - 16)]
    return dict(x=x, y=y, z=z, eps=e, npml=[8, 8, 8], periodic=[False] * 3, source=src, monitors=mons,
                lambdas=np.linspace(1.5, 1.6, c["n_lambda"]), maxTime=c["steps"] * S, shutoff=0.0, precision=c["precision"])


def _serve_jobs(c, seed, ctx):
    """A few 2D couplers and unit cells of uneven size: (dims, sim) in arrival order."""
    r = np.random.default_rng(seed)
    size = np.random.default_rng(2000 + c["n"])
    jobs = []
    for q in range(c["n"]):
        if q % 4 == 3:
            jobs.append((3, _cell_sim(dict(c, nx=int(size.integers(20, 60)), ny=int(size.integers(20, 60)),
                                           nz=int(size.integers(110, 180))), seed + q, ctx)))
        else:
            jobs.append((2, _coupler_sim(dict(c, nx=int(size.integers(450, 1400)), nz=int(size.integers(230, 420))), r)))
    return jobs


def _fdfd_problem(c, seed):
    """An SOI slab with a scattered set of silicon blocks; a line current, a
    second current and an adjoint source (20 nm grid, 30-cell layers)."""
    r = np.random.default_rng(seed)
    d, nx, nz = 0.02, c["nx"], c["nz"]
    x, z = np.arange(nx) * d, np.arange(nz) * d
    zc = 0.55 * nz * d
    boxes = [[-np.inf, np.inf, zc - 0.11, zc + 0.11, N_SI]]
    for _ in range(20):
        a, b = r.uniform(0.3, 0.7) * nx * d, r.uniform(0.35, 0.75) * nz * d
        boxes.append([a, a + r.uniform(0.05, 0.3), b, b + r.uniform(0.05, 0.3), N_SI])
    eps = epsFromBoxes(x, z, N_OX, np.array(boxes))
    f = np.exp(-((z - zc) / 0.15) ** 2)
    J = np.zeros((nx, nz))
    J[nx // 4] = f
    J2 = np.zeros((nx, nz))
    J2[3 * nx // 4] = f * r.uniform(0.5, 1.5)
    g = np.zeros((nx, nz), dtype=np.complex128)
    g[2 * nx // 3] = f * np.exp(1j * r.uniform(0, 6, nz))
    return dict(x=x, z=z, eps=eps, lam=1.55, J=J, J2=J2, g=g)


def _sims(case, seed, ctx):
    """[(dims, sim)] of a time-domain case."""
    k = case["kind"]
    r = np.random.default_rng(seed)
    if k == "slab":
        return [(2, _slab_sim(case, seed))]
    if k == "coupler":
        return [(2, _coupler_sim(case, r))]
    if k in ("pixel", "pixel_call"):
        return [(2, _pixel_sim(case, seed))]
    if k == "batch":
        return [(2, s) for s in _batch_sims(case, seed)]
    if k in ("pillar", "pillar_call"):
        return [(3, _pillar_sim(case, seed, ctx))]
    if k == "cell":
        return [(3, _cell_sim(case, seed, ctx))]
    if k == "strip":
        return [(3, _strip_sim(case, seed))]
    return _serve_jobs(case, seed, ctx)


def prepare(case: dict, seed: int) -> dict:
    ctx = Context(0)
    k = case["kind"]
    if k in ("fdfd", "fdfd_solves"):
        p = _fdfd_problem(case, seed)
        st = dict(kind=k, ctx=ctx, p=p)
        if k == "fdfd_solves":   # the factors that an optimiser keeps for its solves
            st["F"] = fdfd2D(p["x"], p["z"], p["eps"], p["lam"], p["J"], ctx=ctx)
        return st
    sims = _sims(case, seed, ctx)
    st = dict(kind=k, ctx=ctx, sims=sims, steps=case["steps"])
    if k in ("pixel", "pillar"):   # a device-resident job, kept from run to run
        st["job"] = Job(sims[0][1], ctx, dims=sims[0][0])
        del st["sims"]
    return st


# -------------------------------------------------------------------- runs --
def _results(outs) -> dict:
    """The numbers of out structs, those of several jobs joined by name."""
    got: dict = {}
    for o in outs:
        if "mon" in o:
            got.setdefault("flux3d", []).append(o["flux"])
            for m in o["mon"]:
                for k in ("Ea", "Eb", "Ha", "Hb"):
                    got.setdefault(k, []).append(m[k])
        else:
            for k in ("flux", "fluxZ", "P", "B", "PZ", "AZ"):
                got.setdefault(k, []).append(o[k])
    return {k: v[0] if len(v) == 1 else np.concatenate([a.ravel(order="F") for a in v]) for k, v in got.items()}


def run(state: dict):
    k, ctx = state["kind"], state["ctx"]
    if k == "fdfd":
        p = state["p"]
        F = fdfd2D(p["x"], p["z"], p["eps"], p["lam"], p["J"], ctx=ctx)
        E = F.E
        F.close()
        return E
    if k == "fdfd_solves":
        p, F = state["p"], state["F"]
        return {"E": F.solve(p["J2"]), "lam": F.adjoint(p["g"])}
    if k in ("pixel", "pillar"):
        job = state["job"]
        job.reset()
        job.advance(state["steps"])
        return _results([job.finish()])
    sims = state["sims"]
    if k == "batch":
        return _results(fdtd2D_batch([s for _, s in sims], ctx))
    if k == "serve":
        srv = Server(ctx)
        tickets = [srv.submit(s, dims) for dims, s in sims]
        srv.drain()
        outs = [srv.result(t) for t in tickets]
        srv.close()
        return _results(outs)
    dims, sim = sims[0]
    return _results([fdtd2D(sim, ctx) if dims == 2 else fdtd3D(sim, ctx)])


# -------------------------------------------------------------------- work --
def _shapes(case):
    """(dims, nx, ny, nz) of every job of a time-domain case."""
    k = case["kind"]
    if k == "batch":
        size = np.random.default_rng(1000 + case["n"])
        return [(2, int(size.integers(600, 1201)), 1, int(size.integers(250, 351))) for _ in range(case["n"])]
    if k == "serve":
        size, got = np.random.default_rng(2000 + case["n"]), []
        for q in range(case["n"]):
            if q % 4 == 3:
                nx, ny = int(size.integers(20, 60)), int(size.integers(20, 60))
                got.append((3, nx, ny, int(size.integers(110, 180))))
            else:
                nx = int(size.integers(450, 1400))
                got.append((2, nx, 1, int(size.integers(230, 420))))
        return got
    if k in ("pillar", "pillar_call", "cell", "strip"):
        return [(3, case["nx"], case["ny"], case["nz"])]
    return [(2, case["nx"], 1, case["nz"])]


def work(case: dict) -> dict:
    """Each permittivity read once and each result written once; the
    operations of the plain update of every cell and step (11 in 2D, 30 in
    3D).  The frequency-domain solver: the operator and currents in, the
    fields out; 8 real operations for each of the 10 N^1.5 complex
    multiply-adds of a nested-dissection factorisation, or of the 16 N log2 N
    of a solve."""
    if case["kind"] in ("fdfd", "fdfd_solves"):
        N = case["nx"] * case["nz"]
        if case["kind"] == "fdfd":
            return {"bytes": 48.0 * N, "flops": 80.0 * N ** 1.5}
        return {"bytes": 64.0 * N, "flops": 2 * 128.0 * N * math.log2(N)}
    nb = fl = 0.0
    lines = 5 if case["kind"] not in ("slab", "cell") else 2
    for dims, nx, ny, nz in _shapes(case):
        cells = nx * ny * nz
        tm = case["kind"] in ("pixel", "pixel_call")
        if case["kind"] not in ("pixel", "pillar"):   # a kept job holds its material index
            nb += 8.0 * cells * (3 if dims == 3 else (2 if tm else 1))
        else:
            nb += 1.0 * cells * (3 if dims == 3 else 2)
        out = 4 * nx * ny if dims == 3 else 2 * max(nx, nz)
        nb += 16.0 * out * case["n_lambda"] * lines
        fl += (30.0 if dims == 3 else 11.0) * cells * case["steps"]
    return {"bytes": nb, "flops": fl}


# ------------------------------------------------- the results in 64 bits --
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _pulse(src, t):
    k0 = 2 * math.pi / src["lambda0"]
    tau = 2 / (src["bw"] * k0)
    t0 = 5 * tau
    if t < 0 or t > 2 * t0:
        return 0.0
    u = (t - t0) / tau
    return math.exp(-u * u) * math.sin(k0 * (t - t0))


def _pml(n, npml, off, dx, S):
    """(b, a) of the recursion psi <- b psi + a d at the n points u = i + off."""
    u = np.arange(n) + off
    b, a = np.ones(n), np.zeros(n)
    if npml > 0:
        depth = np.where(u < npml, npml - u, np.where(u > n - 1 - npml, u - (n - 1 - npml), 0.0))
        sig = 0.8 * 4.0 / dx * np.minimum(depth / npml, 1.0) ** 3
        on = depth > 0
        b[on] = np.exp(-sig[on] * S)
        a[on] = b[on] - 1.0
    return torch.tensor(b, device=_dev()), torch.tensor(a, device=_dev())


class _Dft:
    """Running transforms of recorded lines: sum_n S exp(i w t_n) x_n."""

    def __init__(self, lambdas, S, off):
        self.w = 2 * math.pi / torch.tensor(np.asarray(lambdas, dtype=float).ravel(), device=_dev())
        self.S, self.off, self.rows, self.t, self.acc = S, off, [], [], None

    def add(self, n, v):
        self.rows.append(v.reshape(-1).clone())
        self.t.append((n + self.off) * self.S)
        if len(self.rows) >= 64:
            self.flush()

    def flush(self):
        if not self.rows:
            return
        x = torch.stack(self.rows)
        ph = self.w[:, None] * torch.tensor(self.t, dtype=torch.float64, device=x.device)[None, :]
        got = torch.complex((torch.cos(ph) * self.S) @ x, (torch.sin(ph) * self.S) @ x)
        self.acc = got if self.acc is None else self.acc + got
        self.rows, self.t = [], []

    def result(self):
        self.flush()
        return self.acc.cpu().numpy()


def _exact2d(sim) -> dict:
    dev, te, per = _dev(), sim["pol"] == "TE", bool(sim.get("periodicZ", False))
    nx, nz = len(sim["x"]), len(sim["z"])
    dx = float(sim["x"][1] - sim["x"][0])
    C = 0.99 / math.sqrt(2)
    S = C * dx
    npx, npz = sim["npml"][0], 0 if per else sim["npml"][1]
    T = lambda v: torch.tensor(np.ascontiguousarray(np.asarray(v).T), device=dev)   # noqa: E731 - [nz][nx]
    cP, cA, cB = (C / T(sim["eps"]), C, C) if te else (C, C / T(sim["epsX"]), C / T(sim["epsZ"]))
    P = torch.zeros(nz, nx, dtype=torch.float64, device=dev)
    nA = nz if per else nz - 1
    A, B = torch.zeros(nA, nx, dtype=P.dtype, device=dev), torch.zeros(nz, nx - 1, dtype=P.dtype, device=dev)
    src = sim["source"]
    s0 = src["ix"] - 1
    f = torch.tensor(np.asarray(src["profile"], dtype=float).ravel(), device=dev)
    srcB = f * (cB if te else cB[:, s0 - 1])
    srcP = f * src["neff"] * (cP[:, s0] if te else cP / T(sim["epsZ"])[:, s0 - 1])
    # one (b, a, psi) per derivative, kept on the two layers of its axis only
    ends = {}

    def layers(key, n, np_, off, axis, shape):
        b, a = _pml(n, np_, off, dx, S)
        got = []
        if np_ > 0:
            last = shape[axis]
            for sl in (slice(0, np_ + 1), slice(last - np_ - 1, last)):
                v = [sl, slice(None)] if axis == 0 else [slice(None), sl]
                bb, aa = (b[sl][:, None], a[sl][:, None]) if axis == 0 else (b[sl][None, :], a[sl][None, :])
                got.append((tuple(v), bb, aa, torch.zeros(shape, dtype=P.dtype, device=dev)[tuple(v)].clone()))
        ends[key] = got

    layers("A", nz, npz, 0.5, 0, (nA, nx))
    layers("B", nx, npx, 0.5, 1, (nz, nx - 1))
    layers("Pz", nz, npz, 0.0, 0, (nz, nx))
    layers("Px", nx, npx, 0.0, 1, (nz, nx))

    def stretch(key, d):
        for sl, b, a, psi in ends[key]:
            psi.mul_(b).add_(a * d[sl])
            d[sl] += psi
        return d

    mons = [int(m) - 1 for m in np.atleast_1d(sim.get("monitors", []))]
    monz = [int(m) - 1 for m in np.atleast_1d(sim.get("monitorsZ", []))]
    lam = sim["lambdas"]
    dP, dB = [_Dft(lam, S, 1.0) for _ in mons], [_Dft(lam, S, 0.5) for _ in mons]
    dPZ, dAZ = [_Dft(lam, S, 1.0) for _ in monz], [_Dft(lam, S, 0.5) for _ in monz]
    zr, zc = torch.zeros(1, nx, dtype=P.dtype, device=dev), torch.zeros(nz, 1, dtype=P.dtype, device=dev)
    for n in range(max(0, math.ceil(sim["maxTime"] / S - 1e-9))):
        gE, gH = _pulse(src, n * S), _pulse(src, (n + 0.5) * S + src["neff"] * 0.5 * dx)
        d = stretch("A", (torch.roll(P, -1, 0) - P) if per else P[1:] - P[:-1])
        A += cA * d
        B -= cB * stretch("B", P[:, 1:] - P[:, :-1])
        B[:, s0 - 1] += srcB * gE
        da = (A - torch.roll(A, 1, 0)) if per else torch.cat((A, zr)) - torch.cat((zr, A))
        db = torch.cat((B, zc), 1) - torch.cat((zc, B), 1)
        P += cP * (stretch("Pz", da) - stretch("Px", db))
        P[:, s0] += srcP * gH
        for q, m in enumerate(mons):
            dP[q].add(n, P[:, m])
            dB[q].add(n, 0.5 * (B[:, m - 1] + B[:, m]))
        for q, m in enumerate(monz):
            dPZ[q].add(n, P[m])
            dAZ[q].add(n, 0.5 * (A[m - 1] + A[m]))
    out = {}
    nL = np.asarray(lam).size
    stack = lambda ds, ln: (np.asfortranarray(np.stack([q.result().T for q in ds], axis=2)) if ds   # noqa: E731
                            else np.zeros((ln, nL, 0), dtype=np.complex128))
    out["P"], out["B"], out["PZ"], out["AZ"] = stack(dP, nz), stack(dB, nz), stack(dPZ, nx), stack(dAZ, nx)
    out["flux"] = 0.5 * dx * np.sum((out["P"] * out["B"].conj()).real, axis=0).T
    out["fluxZ"] = -0.5 * dx * np.sum((out["PZ"] * out["AZ"].conj()).real, axis=0).T
    return out


def _exact3d(sim) -> dict:
    dev, per = _dev(), [bool(v) for v in sim["periodic"]]
    n = [len(sim[k]) for k in "xyz"]
    d = float(sim["x"][1] - sim["x"][0])
    C = 0.99 / math.sqrt(3)
    S = C * d
    shape = (n[2], n[1], n[0])
    ax = lambda q: 2 - q   # noqa: E731 - tensor axis of x, y, z
    T = lambda v: torch.tensor(np.ascontiguousarray(np.asarray(v).T), device=dev)   # noqa: E731
    cE = [C / T(sim["eps"][k]) for k in "xyz"]
    E = [torch.zeros(shape, dtype=torch.float64, device=dev) for _ in range(3)]
    H = [torch.zeros(shape, dtype=torch.float64, device=dev) for _ in range(3)]
    npml = [0 if per[q] else int(sim["npml"][q]) for q in range(3)]
    psi = {}
    for q in range(3):
        for kind, off in (("H", 0.5), ("E", 0.0)):
            b, a = _pml(n[q], npml[q], off, d, S)
            if npml[q] == 0:
                continue
            for c in range(3):
                if c == q:
                    continue
                got = []
                for sl in (slice(0, npml[q] + 1), slice(n[q] - npml[q] - 1, n[q])):
                    v = [slice(None)] * 3
                    v[ax(q)] = sl
                    sh = [1, 1, 1]
                    sh[ax(q)] = -1
                    full = list(shape)
                    full[ax(q)] = npml[q] + 1
                    got.append((tuple(v), b[sl].reshape(sh), a[sl].reshape(sh), torch.zeros(full, dtype=E[0].dtype, device=dev)))
                psi[kind, c, q] = got

    def diff(F, q, kind, c):
        a = ax(q)
        if kind == "H":
            g = torch.roll(F, -1, a) - F
            if not per[q]:
                v = [slice(None)] * 3
                v[a] = n[q] - 1
                g[tuple(v)] = -F[tuple(v)]
        else:
            g = F - torch.roll(F, 1, a)
            if not per[q]:
                v = [slice(None)] * 3
                v[a] = 0
                g[tuple(v)] = F[tuple(v)]
        for sl, b, aa, ps in psi.get((kind, c, q), []):
            ps.mul_(b).add_(aa * g[sl])
            g[sl] += ps
        return g

    src = sim["source"]
    sa = src["axis"] - 1
    sb, sc = (sa + 1) % 3, (sa + 2) % 3
    ss = src["index"] - 1

    def at(q, i):
        v = [slice(None)] * 3
        v[ax(q)] = i
        return tuple(v)

    def plane(v):
        """A profile [n_b][n_c] (or a number) laid out as a plane normal to sa."""
        if np.ndim(v) == 0:
            return float(v)
        t = torch.tensor(np.asarray(v, dtype=float), device=dev)
        return t.T if ax(sb) > ax(sc) else t

    Ea, Eb, Ha, Hb = (plane(src[k]) for k in ("Ea", "Eb", "Ha", "Hb"))
    lam = sim["lambdas"]
    mons = [(m["axis"] - 1, m["index"] - 1) for m in sim["monitors"]]
    dft = [[_Dft(lam, S, 1.0 if k < 2 else 0.5) for k in range(4)] for _ in mons]
    for s in range(max(0, math.ceil(sim["maxTime"] / S - 1e-9))):
        gE, gH = _pulse(src, s * S), _pulse(src, (s + 0.5) * S + src["neff"] * 0.5 * d)
        for c in range(3):
            c1, c2 = (c + 1) % 3, (c + 2) % 3
            H[c] -= C * (diff(E[c2], c1, "H", c) - diff(E[c1], c2, "H", c))
        H[sb][at(sa, ss - 1)] -= C * Eb * gE
        H[sc][at(sa, ss - 1)] += C * Ea * gE
        for c in range(3):
            c1, c2 = (c + 1) % 3, (c + 2) % 3
            E[c] += cE[c] * (diff(H[c2], c1, "E", c) - diff(H[c1], c2, "E", c))
        E[sb][at(sa, ss)] += cE[sb][at(sa, ss)] * (Hb * gH)
        E[sc][at(sa, ss)] -= cE[sc][at(sa, ss)] * (Ha * gH)
        for (q, i), D in zip(mons, dft):
            qa, qb = (q + 1) % 3, (q + 2) % 3
            for F, t in ((E[qa], D[0]), (E[qb], D[1])):
                v = F[at(q, i)]
                t.add(s, v if ax(qa) > ax(qb) else v.T)
            for F, t in ((H[qa], D[2]), (H[qb], D[3])):
                v = 0.5 * (F[at(q, i)] + F[at(q, i - 1)])
                t.add(s, v if ax(qa) > ax(qb) else v.T)
    out = {"mon": [], "flux": np.zeros((len(mons), np.asarray(lam).size))}
    for k, ((q, _), D) in enumerate(zip(mons, dft)):
        na, nb = n[(q + 1) % 3], n[(q + 2) % 3]
        # rows run over (b, a), a fastest: back to [a][b][lambda]
        m = {key: np.asfortranarray(t.result().reshape(-1, nb, na).transpose(2, 1, 0))
             for key, t in zip(("Ea", "Eb", "Ha", "Hb"), D)}
        out["mon"].append(m)
        out["flux"][k] = 0.5 * d * d * np.sum((m["Ea"] * m["Hb"].conj() - m["Eb"] * m["Ha"].conj()).real, axis=(0, 1))
    return out


def _exact_fdfd(p, rhs) -> list:
    """Block elimination of the five-point operator along x in complex 128-bit
    arithmetic: solutions of A E = v (or A.' E = v) for rhs = [(v, transposed)]."""
    dev = _dev()
    nx, nz = p["eps"].shape
    d, k0, npml, R = float(p["x"][1] - p["x"][0]), 2 * math.pi / p["lam"], 30, 1e-8

    def s(n, half):
        u = np.arange(n + 1) - 0.5 if half else np.arange(n, dtype=float)
        L = npml * d
        depth = np.where(u < npml, npml - u, np.where(u > n - 1 - npml, u - (n - 1 - npml), 0.0)) * d
        return 1 + 2j * math.log(1 / R) / (k0 * L) * (depth / L) ** 3

    sx, sxh, sz, szh = s(nx, False), s(nx, True), s(nz, False), s(nz, True)
    xm, xp = 1 / (d * d * sx * sxh[:-1]), 1 / (d * d * sx * sxh[1:])
    zm, zp = 1 / (d * d * sz * szh[:-1]), 1 / (d * d * sz * szh[1:])
    t = lambda v: torch.tensor(np.asarray(v, dtype=np.complex128), device=dev)   # noqa: E731
    Z = t(np.diag(zm[1:], -1) + np.diag(zp[:-1], 1))
    diag = t(-(xm + xp)[:, None] - (zm + zp)[None, :] + k0 * k0 * p["eps"])
    got = []
    inv = []
    for i in range(nx):
        D = Z + torch.diag(diag[i])
        if i:
            D = D - complex(xm[i]) * complex(xp[i - 1]) * inv[-1]
        inv.append(torch.linalg.inv(D))
    for v, tr in rhs:
        v = t(v)
        lo, up = (xm, xp) if not tr else (np.roll(xp, 1), np.roll(xm, -1))   # rows' couplings to i - 1, i + 1
        y = []
        for i in range(nx):
            w = v[i] - (complex(lo[i]) * y[-1] if i else 0)
            y.append((inv[i].T if tr else inv[i]) @ w)
        e = [None] * nx
        e[-1] = y[-1]
        for i in range(nx - 2, -1, -1):
            e[i] = y[i] - (inv[i].T if tr else inv[i]) @ (complex(up[i]) * e[i + 1])
        got.append(torch.stack(e).cpu().numpy())
    return got


def exact(case: dict, seed: int):
    k = case["kind"]
    if k == "fdfd":
        p = _fdfd_problem(case, seed)
        return _exact_fdfd(p, [(-p["J"], False)])[0]
    if k == "fdfd_solves":
        p = _fdfd_problem(case, seed)
        E, lam = _exact_fdfd(p, [(-p["J2"], False), (p["g"], True)])
        return {"E": E, "lam": lam}
    if k == "batch":
        return None   # many runs one after the other: too long here, and the single couplers stand for them
    sims = _sims(case, seed, Context(0) if torch.cuda.is_available() else None)
    return _results([_exact2d(s) if dims == 2 else _exact3d(s) for dims, s in sims])
