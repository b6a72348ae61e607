"""The work this library is run for, as cases that can be timed and checked: time steps of the shipped physics from
host states, on static, batched and moving clouds, in both precisions, with the set-up of a cloud where that is part of
the work. Every pass goes through the public entry points (Context / GB300RKTimeStepper over the C ABI) from the
caller's own host arrays to the advanced state in the caller's own host array, so it can be repeated.

Each step takes its dt from the CFL call, as the reference's time loop does. FP32 states are smooth (random Fourier
modes): the MOOD checks and their fixed points run on the extrema of every field, and a particle whose candidate sits
on the edge of a bound changes the result by the smooth fields' truncation error only. FP64 states have jumps.

`exact` restates the methods in 64 bits with torch operations over the list of neighbour pairs."""
import dataclasses
import importlib.util
import math
import sys
from functools import lru_cache
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
GAMMA = 1.4
RING = [(math.cos(2 * math.pi * q / 16), math.sin(2 * math.pi * q / 16)) for q in range(16)]
BGK = dict(epsilon=1e-4, macro_velocity=(1.0, 0.5))
ADVECTION = ((1.0,), (0.5,))


def package():
    if "hcc_gb300" not in sys.modules:
        pkg = ROOT / "hypercloudcore.jl_gb300"
        spec = importlib.util.spec_from_file_location("hcc_gb300", pkg / "__init__.py",
                                                      submodule_search_locations=[str(pkg)])
        sys.modules["hcc_gb300"] = mod = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(mod)
    return sys.modules["hcc_gb300"]


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest call: the reference's plain 2-D advection run (FP64, MUSCL2 + MOOD) on a cloud of a few
        # thousand points, where launches and latency count
        {"name": "advection2d_fp64_small", "kind": "advection", "precision": "fp64", "nx": 50, "ny": 47, "steps": 4},
        # the reference's published benchmark case: third order, Venkatakrishnan limiter, periodic, both precisions
        {"name": "advection2d_order3_fp32", "kind": "advection3", "precision": "fp32", "nx": 1000, "ny": 1000, "steps": 4},
        {"name": "advection2d_order3_fp64", "kind": "advection3", "precision": "fp64", "nx": 301, "ny": 250, "steps": 2},
        # 2-D Euler at the configured 1M nodes in the FP32 bulk path
        {"name": "euler2d_fp32", "kind": "euler", "dim": 2, "precision": "fp32", "nx": 1000, "ny": 1000, "steps": 4},
        # 2-D Euler in the plain FP64 path from a Voronoi Riemann state: the MOOD fixed points at jumps
        {"name": "euler2d_fp64", "kind": "euler", "dim": 2, "precision": "fp64", "nx": 256, "ny": 251, "steps": 2},
        # 3-D Euler FP32: a small ragged box (a tile or two per SM), and the bulk case at 1.3M interior points
        {"name": "euler3d_fp32_small", "kind": "euler", "dim": 3, "precision": "fp32", "nx": 33, "ny": 29, "nz": 31, "steps": 4},
        {"name": "euler3d_fp32", "kind": "euler", "dim": 3, "precision": "fp32", "nx": 110, "ny": 110, "nz": 110, "steps": 2},
        # 3-D Euler in the plain FP64 path from a spherical blast
        {"name": "euler3d_fp64", "kind": "euler", "dim": 3, "precision": "fp64", "nx": 41, "ny": 40, "nz": 40, "steps": 1},
        # the batched ensemble of uneven kinetic-relaxation clouds (16 velocities, IMEX), one dt per cloud
        {"name": "bgk_batch_fp32", "kind": "bgk", "precision": "fp32", "clouds": 24, "largest": 128000, "steps": 2},
        # the meshless-WENO variant of 3-D Euler
        {"name": "weno3d_fp32", "kind": "weno", "dim": 3, "precision": "fp32", "nx": 48, "ny": 48, "nz": 45, "steps": 1},
        # a new stepper on a new cloud and its first step: neighbour search, MLS geometry and tables
        {"name": "setup3d_fp32", "kind": "setup", "dim": 3, "precision": "fp32", "nx": 64, "ny": 64, "nz": 64, "steps": 1},
        # a Lagrangian run on a moving cloud: the geometry refreshed at every stage, a search after every step
        {"name": "moving2d_fp64", "kind": "moving", "dim": 2, "precision": "fp64", "nx": 128, "ny": 120, "steps": 3},
    ]


def draw(rng):
    """One more case: a kind, a precision and log-uniform sizes with ragged sides."""
    kind = rng.choice(["advection", "advection3", "euler", "euler", "euler", "bgk", "weno", "setup", "moving"])
    prec = rng.choice(["fp32", "fp64"])
    dim = rng.choice([2, 3])

    def sides(lo, hi, d):
        n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        s = [max(9, round(n ** (1 / d) * rng.uniform(0.9, 1.1))) for _ in range(d)]
        return dict(zip(("nx", "ny", "nz"), s))

    if kind == "advection":
        return {"kind": kind, "precision": prec, **sides(1.5e3, 5e5, 2), "steps": rng.randint(2, 4)}
    if kind == "advection3":
        return {"kind": kind, "precision": prec, **sides(1e4, 8e5 if prec == "fp32" else 1e5, 2), "steps": rng.randint(1, 4)}
    if kind == "bgk":
        return {"kind": kind, "precision": "fp32", "clouds": rng.randint(3, 24),
                "largest": round(math.exp(rng.uniform(math.log(8e3), math.log(1.2e5)))), "steps": rng.randint(1, 2)}
    if kind == "weno":
        n = (1.5e4, 9e4) if prec == "fp32" else (3e3, 9e3)
        return {"kind": kind, "dim": 3, "precision": prec, **sides(*n, 3), "steps": 1}
    if kind == "setup":
        return {"kind": kind, "dim": dim, "precision": prec, **sides(1e4, 2e5 if prec == "fp32" else 4e4, dim), "steps": 1}
    if kind == "moving":
        return {"kind": kind, "dim": 2, "precision": prec, **sides(3e3, 4e4, 2), "steps": rng.randint(1, 3)}
    hi = {(2, "fp32"): 9e5, (3, "fp32"): 7e5, (2, "fp64"): 9e4, (3, "fp64"): 6e4}[(dim, prec)]
    return {"kind": kind, "dim": dim, "precision": prec, **sides(5e3, hi, dim), "steps": rng.randint(1, 4 if prec == "fp32" else 2)}


# ------------------------------------------------------------------------------------------------ inputs
def sizes(case):
    return [case[k] for k in ("nx", "ny", "nz") if k in case]


@lru_cache(maxsize=4)
def box_cloud(n, periodic, jittered, seed):
    """A lattice of spacing 1/n[0] over a box of n cells, jittered by a quarter cell, with its ghost band."""
    h = 1.0 / n[0]
    return package().rectangular_cloud((0.0,) * len(n), tuple(k * h for k in n), h, 2.5 * h, periodic=periodic,
                                       jitter=0.25 * h if jittered else None, seed=seed)


def shaken(cloud, rng):
    """The cloud with the points away from the walls moved a little: new positions, the same number and tags."""
    h, pos = cloud.dx[0], cloud.pos.copy()
    free = ((pos > np.array(cloud.domain_min) + h) & (pos < np.array(cloud.domain_max) - h)).all(axis=1)
    pos[free] += 0.05 * h * rng.uniform(-1, 1, (int(free.sum()), cloud.dim))
    return dataclasses.replace(cloud, pos=pos)


@lru_cache(maxsize=2)
def batch_clouds(count, largest):
    """Square clouds with log-uniform node counts up to `largest`, one spacing."""
    rng, h = np.random.default_rng(2026), 1.0 / 256
    n = np.exp(rng.uniform(math.log(4000.0), math.log(largest), count - 1)).tolist() + [largest]
    side = [max(8, round(math.sqrt(k)) - 1) for k in n]
    return tuple(package().rectangular_cloud((0.0, 0.0), (s * h, s * h), h, 2.5 * h, jitter=0.25 * h, seed=1000 + k)
                 for k, s in enumerate(side))


def waves(x, rng, amplitude, modes=3, top=2):
    """A smooth random field over the unit box: a few low Fourier modes, |value| <= amplitude."""
    f = np.zeros(len(x))
    for _ in range(modes):
        k = rng.integers(-top, top + 1, x.shape[1])
        k[rng.integers(x.shape[1])] = rng.integers(1, top + 1)
        f += rng.uniform(0.5, 1.0) * np.sin(2 * math.pi * (x @ k) + rng.uniform(0, 2 * math.pi))
    return (amplitude / modes) * f


def conserved(rho, u, p):
    return np.column_stack([rho] + [rho * v for v in u] + [p / (GAMMA - 1) + 0.5 * rho * sum(v * v for v in u)])


def euler_state(cloud, rng, smooth):
    ext = np.array(cloud.domain_max) - np.array(cloud.domain_min)
    x, D = (cloud.pos - np.array(cloud.domain_min)) / ext, cloud.dim
    if smooth:
        return conserved(1 + waves(x, rng, 0.4), [waves(x, rng, 0.4) for _ in range(D)], 1 + waves(x, rng, 0.4))
    if D == 2:   # random Voronoi regions
        k = int(rng.integers(2, 7))
        r = np.argmin(((x[:, None, :] - rng.random((k, 2))[None]) ** 2).sum(axis=2), axis=1)
        rho, p, u, v = (rng.uniform(a, b, k)[r] for a, b in ((0.1, 2), (0.1, 2), (-1, 1), (-1, 1)))
        return conserved(rho, [u, v], p)
    inside = ((x - rng.uniform(0.4, 0.6, 3)) ** 2).sum(axis=1) < rng.uniform(0.18, 0.25) ** 2
    return conserved(np.where(inside, 1.0, 0.125), [np.zeros(len(x))] * 3, np.where(inside, 1.0, 0.1))


def kinetic():
    return package().KineticRelaxation(RING, **BGK)


def make_inputs(case, seed):
    """(cloud or clouds, U0, what make_config needs) of a case: host arrays."""
    hcc, rng, kind = package(), np.random.default_rng(seed), case["kind"]
    f32 = case["precision"] == "fp32"
    if kind == "bgk":
        cloud = batch_clouds(case["clouds"], case["largest"])
        h = cloud[0].dx[0]
        ext = [np.array(c.domain_max) for c in cloud]
        U0 = np.concatenate([kinetic().maxwellian(1 + waves(c.pos / e, rng, 0.3)) for c, e in zip(cloud, ext)])
        spec = dict(pde=kinetic(), scheme=hcc.MUSCL(2, 2), mood=hcc.MOOD(hcc.EPD1, hcc.MOODu1(1e-4 * h * h)),
                    tableau="IMEX_ARS222", bc_map={t: hcc.BC_OUTFLOW for t in range(1, 5)})
        return cloud, np.ascontiguousarray(U0, dtype=np.float32), spec
    n = tuple(sizes(case))
    D, h = len(n), 1.0 / n[0]
    cloud = box_cloud(n, kind in ("advection3", "moving"), kind != "advection3", 42)
    if kind in ("setup", "moving"):            # the cloud itself is what is new
        cloud = shaken(cloud, rng)
    spec = dict(scheme=hcc.MUSCL(2, 2), mood=hcc.MOOD(hcc.EPD1, hcc.MOODu1(1e-4 * h ** D)), tableau="RK3_SSP")
    if kind == "advection":
        c = rng.uniform(0.25, 0.4, 2)
        U0 = np.exp(-((cloud.pos - c) ** 2).sum(axis=1) / 0.02)[:, None] * rng.uniform(0.8, 1.2)
        spec.update(pde=hcc.LinearAdvection(ADVECTION), bc_map={1: hcc.BC_DIRICHLET, 2: hcc.BC_OUTFLOW,
                                                                3: hcc.BC_DIRICHLET, 4: hcc.BC_OUTFLOW})
    elif kind == "advection3":
        x = cloud.pos / np.array(cloud.domain_max)
        U0 = (1 + np.exp(-((x - rng.uniform(0.45, 0.55, 2)) ** 2).sum(axis=1) / 0.02) + waves(x, rng, 0.2))[:, None]
        spec.update(pde=hcc.LinearAdvection(ADVECTION), scheme=hcc.MUSCL(3, 0, "vk_hard"),
                    mood=hcc.MOOD(hcc.EPD1, hcc.MOODu1(1e-6)))
    else:
        U0 = euler_state(cloud, rng, f32 or kind == "moving")
        spec.update(pde=hcc.Euler(D, GAMMA), bc_map={t: hcc.BC_OUTFLOW for t in range(1, 2 * D + 1)})
        if kind == "weno":
            spec["scheme"] = hcc.WENO(2)
    return cloud, np.ascontiguousarray(U0, dtype=np.float32 if f32 else np.float64), spec


def cfl_of(case):
    return 0.3 if case["kind"] == "advection3" else 0.4


class State:
    pass


def pinned(shape, dtype):
    t = {np.dtype(np.float32): torch.float32, np.dtype(np.float64): torch.float64}[np.dtype(dtype)]
    return torch.empty(shape, dtype=t, pin_memory=torch.cuda.is_available()).numpy()


def prepare(case, seed):
    hcc, s = package(), State()
    s.case = case
    s.cloud, U0, s.spec = make_inputs(case, seed)
    s.U0, s.out = pinned(U0.shape, U0.dtype), pinned(U0.shape, U0.dtype)
    s.U0[:] = U0
    if case["kind"] == "setup":
        return s
    first = s.cloud[0] if case["kind"] == "bgk" else s.cloud
    pde = s.spec.pop("pde")
    s.ctx = hcc.Context(hcc.make_config(pde, first, precision=case["precision"], **s.spec))
    if case["kind"] == "moving":
        s.ctx.set_mover(hcc.mover("lagrangian"))
        return s
    if case["kind"] == "bgk":
        s.ctx.upload_batch(s.cloud)
    else:
        s.ctx.upload_cloud(s.cloud)
    s.ctx.build_neighbours()
    s.ctx.prepare_geometry()
    return s


def run(s):
    case, cfl, t = s.case, cfl_of(s.case), 0.0
    if case["kind"] == "setup":
        spec = dict(s.spec)
        ts = package().GB300RKTimeStepper(spec.pop("pde"), s.cloud, precision=case["precision"], **spec)
        ts.set_state(s.U0)
        dt = cfl * ts.get_time_step()
        ts(t, dt)
        ts.ctx.download_state(out=s.out)
        ts.ctx.close()
        return {"U": s.out, "t": np.float64(dt) if s.U0.dtype == np.float64 else np.float32(dt)}
    ctx = s.ctx
    if case["kind"] == "moving":               # back to the start: the cloud, then its state
        ctx.upload_cloud(s.cloud)
        ctx.build_neighbours()
        ctx.prepare_geometry()
    ctx.upload_state(s.U0)
    if case["kind"] == "bgk":
        t = np.zeros(len(s.cloud))
        for _ in range(case["steps"]):
            dts = cfl * ctx.batch_time_steps()
            ctx.step_batch(0.0, dts)
            t = t + dts
        return {"U": ctx.download_state(out=s.out), "t": t.astype(np.float32)}
    for _ in range(case["steps"]):
        dt = cfl * ctx.time_step()
        ctx.step(t, dt)
        t += dt
    got = {"U": ctx.download_state(out=s.out), "t": np.float64(t) if s.U0.dtype == np.float64 else np.float32(t)}
    if case["kind"] == "moving":
        got["x"], got["V"] = ctx.positions(), ctx.volumes()
        if s.U0.dtype == np.float32:           # the particles follow an FP32 velocity
            got["x"], got["V"] = got["x"].astype(np.float32), got["V"].astype(np.float32)
    return got


def work(case):
    """One pass: per point and stage the neighbour indices, the position and the stage's states once; per slot the
    reconstructions, the fluxes and their contraction."""
    kind, s = case["kind"], 8 if case["precision"] == "fp64" else 4
    if kind == "bgk":
        n, D, M = 0.27 * case["clouds"] * case["largest"], 2, 16
    else:
        n, D = float(np.prod(sizes(case))), len(sizes(case))
        M = 1 if kind.startswith("advection") else D + 2
    K = 19.6 if D == 2 else 65.4
    per_flux = 2 * D * M + 8 * M
    flops = K * (4 * D * M + 2 * per_flux + 6 * M + 2 * M * D) if kind != "weno" else K * D * (8 * M * D + 8 * M)
    nbytes = 3 * case["steps"] * n * (4 * K + 8 * D + 6 * s * M) + 2 * n * s * M
    flops = 3 * case["steps"] * n * flops
    if kind in ("setup", "moving"):            # search, moments and weights of every geometry
        geoms = 1 if kind == "setup" else 1 + 3 * case["steps"]
        nbytes += geoms * n * (K * (4 + 8 * (2 * D + 1)) + 8 * D)
        flops += geoms * n * K * (2 * (D + 1) ** 2 * 3 + 6 * D)
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------------------------------------ 64 bits
def neighbour_pairs(pos, R, length, low, high):
    """(i, j, x_j - x_i) of every ordered pair within R, sorted by i; `length`: the period of each axis or 0."""
    N, D = pos.shape
    dims = [max(1, int((high[d] - low[d]) / (1.0001 * R))) for d in range(D)]
    cart = [((pos[:, d] - low[d]) * (dims[d] / (high[d] - low[d]))).long().clamp(0, dims[d] - 1) for d in range(D)]
    ncell = math.prod(dims)
    lin = sum(c * math.prod(dims[:d]) for d, c in enumerate(cart))
    order = torch.argsort(lin)
    count = torch.bincount(lin, minlength=ncell + 1)
    start = torch.cumsum(count, 0) - count
    got = []
    for off in range(3 ** D):
        cell, ok = torch.zeros_like(lin), torch.ones(N, dtype=torch.bool, device=pos.device)
        for d in range(D):
            c = cart[d] + (off // 3 ** d) % 3 - 1
            if length[d]:
                c = c % dims[d]
            ok &= (c >= 0) & (c < dims[d])
            cell += c * math.prod(dims[:d])
        cell = torch.where(ok, cell, ncell)
        m = count[cell]
        i = torch.repeat_interleave(torch.arange(N, device=pos.device), m)
        j = order[start[cell][i] + torch.arange(len(i), device=pos.device) - (torch.cumsum(m, 0) - m)[i]]
        x = pos[j] - pos[i]
        for d in range(D):
            if length[d]:
                x[:, d] -= length[d] * torch.round(x[:, d] / length[d])
        keep = ((x * x).sum(1) <= R * R) & (i != j)
        got.append((i[keep], j[keep], x[keep]))
    i, j, x = (torch.cat(v) for v in zip(*got))
    s = torch.argsort(i, stable=True)
    return i[s], j[s], x[s]


def taylor(x, degree):
    """The monomials of degree 1..degree over their factorials: first-degree terms first, second-degree ones next."""
    D = x.shape[1]
    cols = [x[:, d] for d in range(D)]
    if degree >= 2:
        cols += [x[:, d] ** 2 / 2 for d in range(D)]
        cols += [x[:, d] * x[:, e] for d in range(D) for e in range(d + 1, D)]
    if degree >= 3:
        cols += [x[:, d] ** 3 / 6 for d in range(D)]
        cols += [x[:, d] ** 2 * x[:, e] / 2 for d in range(D) for e in range(D) if e != d]
        if D == 3:
            cols += [x[:, 0] * x[:, 1] * x[:, 2]]
    return torch.stack(cols, 1)


class Method:
    """The methods over the pairs of one cloud, in 64 bits."""
    PART = 4 << 20                             # pairs handled at a time

    def __init__(self, case, cloud, spec, dev):
        self.case, self.dev, self.D = case, dev, cloud.dim
        self.kind = case["kind"]
        t = lambda a: torch.tensor(np.asarray(a), dtype=torch.float64, device=dev)  # noqa: E731
        self.h, self.R = cloud.dx[0], cloud.radius
        self.low, self.high = list(cloud.canvas_min), list(cloud.canvas_max)
        self.box = [b - a for a, b in zip(cloud.domain_min, cloud.domain_max)]
        self.origin = list(cloud.domain_min)
        self.length = [L if p else 0.0 for L, p in zip(self.box, cloud.periodic)]
        self.bnd = torch.tensor(cloud.is_boundary.astype(bool), device=dev)
        self.tags = torch.tensor(cloud.tags.astype(np.int64), device=dev)
        self.outflow = [tag for tag, kind in (spec.get("bc_map") or {}).items() if kind == package().BC_OUTFLOW]
        self.order = spec["scheme"].order
        self.limited = self.kind == "advection3"
        self.delta = spec["mood"].criterion.delta
        self.pad = 16 * 2.0 ** -23 if case["precision"] == "fp32" else 0.0   # of the FP32 path's bounds
        if spec["tableau"] == "RK3_SSP":
            self.A, self.b = [[0, 0, 0], [1, 0, 0], [0.25, 0.25, 0]], [1 / 6, 1 / 6, 2 / 3]
            self.Ai, self.bi, self.substep = None, None, True
        else:
            g = 1 - 1 / math.sqrt(2)
            d = 1 - 1 / (2 * g)
            self.A, self.b = [[0, 0, 0], [g, 0, 0], [d, 1 - d, 0]], [d, 1 - d, 0]
            self.Ai, self.bi, self.substep = [[0, 0, 0], [0, g, 0], [0, 1 - g, g]], [0, 1 - g, g], False
        self.pde = spec["pde"]
        if self.kind == "bgk":
            self.c = t(RING).T
            self.sinv = torch.where(self.c.T.abs() > 1e-14, self.D / self.c.T, torch.zeros_like(self.c.T))
        elif self.kind.startswith("advection"):
            self.c = t(ADVECTION)
        self.x = t(cloud.pos)
        self.search()

    # ---- geometry
    def search(self):
        for d in range(self.D):
            if self.length[d]:
                self.x[:, d] = self.origin[d] + torch.remainder(self.x[:, d] - self.origin[d], self.length[d])
        self.i, self.j, self.dist = neighbour_pairs(self.x, self.R, self.length, self.low, self.high)
        self.geometry()

    def sum(self, v):
        out = torch.zeros((len(self.x),) + v.shape[1:], dtype=v.dtype, device=v.device)
        return out.index_add_(0, self.i, v)

    def parts(self):
        for a in range(0, len(self.i), self.PART):
            yield slice(a, min(len(self.i), a + self.PART))

    def fit(self, degree, intercept, mask=None):
        """Rows of the inverse moment matrix of the weighted fit at every particle, (N, D or B, B)."""
        B = taylor(self.dist[:1], degree).shape[1] + intercept
        N = torch.zeros((len(self.x), B, B), dtype=torch.float64, device=self.dev)
        for s in self.parts():
            p = self.basis(s, degree, intercept)
            w = self.w[s] if mask is None else self.w[s] * mask[s]
            N.index_add_(0, self.i[s], (w[:, None] * p)[:, :, None] * p[:, None, :])
        eye = torch.eye(B, dtype=torch.float64, device=self.dev)
        bad = self.bnd | (torch.linalg.cholesky_ex(N + 0 * eye)[1] != 0)
        return torch.linalg.inv(torch.where(bad[:, None, None], eye, N)) * (~bad)[:, None, None]

    def basis(self, s, degree, intercept=False):
        p = taylor(self.dist[s] / self.h, degree)
        return torch.cat([torch.ones_like(p[:, :1]), p], 1) if intercept else p

    def slopes(self, degree, intercept, mask=None):
        """Per pair the weights of the first derivatives: sum_k c_k f_k = grad f."""
        inv = self.fit(degree, intercept, mask)
        out = torch.empty_like(self.dist)
        for s in self.parts():
            rows = inv[:, int(intercept):int(intercept) + self.D][self.i[s]]
            out[s] = (rows * self.basis(s, degree, intercept)[:, None, :]).sum(2) * (self.w[s] / self.h)[:, None]
        return out if mask is None else out * mask[:, None]

    def geometry(self):
        r2 = (self.dist * self.dist).sum(1)
        y = r2 / self.R ** 2
        self.w = torch.where(r2 <= self.R ** 2, 1 / (1 + y * (1 + y * (0.5 + y * (1 / 6 + y / 24)))), 0.0)
        self.count = torch.bincount(self.i, minlength=len(self.x))
        if self.kind == "weno":
            self.dw = self.slopes(2, False)
            self.central = {1: self.slopes(1, False), 2: self.dw}
            self.sides = {}
        else:
            self.recon = self.fit(self.order - 1, False)
            self.dw = self.dw_low = self.slopes(1, True)
            if self.order == 3:
                self.recon_low = self.fit(1, False)
                self.dw = self.slopes(3, True)
                few = (2 * self.count < 30)[self.i]
                if bool(few.any()):
                    self.dw = torch.where(few[:, None], self.slopes(2, True), self.dw)
        self.donor = torch.where(self.bnd, -1, torch.arange(len(self.x), device=self.dev))
        for tag in self.outflow:               # the nearest resolved neighbour, in at most five passes
            status = torch.where(self.bnd, torch.where(self.tags == tag, 0, -1), 1)
            for n in range(1, 6):
                ok = (status[self.i] == 0) & (status[self.j] > 0)
                if not bool(ok.any()):
                    break
                i, j, d = self.i[ok], self.j[ok], r2[ok]
                best = torch.full((len(self.x),), math.inf, dtype=torch.float64, device=self.dev)
                best.scatter_reduce_(0, i, d, "amin")
                hit = d == best[i]
                self.donor[i[hit]] = self.donor[j[hit]]
                status[i[hit]] = n + 1

    # ---- physics
    def speed(self, U):
        if not isinstance(self.pde, package().Euler):
            return self.c.abs().amax(1).expand(len(U), self.D)
        u = U[:, 1:-1] / U[:, :1]
        p = (GAMMA - 1) * (U[:, -1] - 0.5 * U[:, 0] * (u * u).sum(1))
        return u.abs() + torch.sqrt(GAMMA * p / U[:, 0])[:, None]

    def flux(self, U, w=None):
        """((n, D, M) fluxes, (n, D) speeds), in the frame of a grid moving with w."""
        if isinstance(self.pde, package().Euler):
            u = U[:, 1:-1] / U[:, :1]
            p = (GAMMA - 1) * (U[:, -1] - 0.5 * U[:, 0] * (u * u).sum(1))
            F = U[:, None, :] * u[:, :, None]
            for d in range(self.D):
                F[:, d, 1 + d] += p
                F[:, d, -1] += p * u[:, d]
            lam = (u if w is None else u - w).abs() + torch.sqrt(GAMMA * p / U[:, 0])[:, None]
            return (F if w is None else F - w[:, :, None] * U[:, None, :]), lam
        return self.c[None] * U[:, None, :], self.c.abs().amax(1).expand(len(U), self.D)

    def time_step(self, U):
        lam, s = self.speed(U), torch.zeros(len(U), dtype=torch.float64, device=self.dev)
        for q in self.parts():
            top = torch.maximum(lam[self.i[q]], lam[self.j[q]])
            s.index_add_(0, self.i[q], (self.dw[q].abs() * top).sum(1))
        return torch.where(self.bnd | (s <= 0), math.inf, 1 / (self.D * s))

    # ---- one right-hand side, at given orders
    def gradients(self, Y, orders):
        M, inv = Y.shape[1], self.recon
        g = torch.zeros((len(Y), inv.shape[1], M), dtype=torch.float64, device=self.dev)
        for s in self.parts():
            v = self.w[s, None] * self.basis(s, self.order - 1)
            g.index_add_(0, self.i[s], v[:, :, None] * (Y[self.j[s]] - Y[self.i[s]])[:, None, :])
        low = None
        if self.order == 3:                    # a particle one order down: the degree-1 fit
            low = torch.zeros_like(g)
            low[:, :self.D] = self.recon_low @ g[:, :self.D]
        g = inv @ g
        if low is not None:
            g = torch.where((orders == 2)[:, None, None], low, g)
        g = g * (orders > 1)[:, None, None]
        if self.limited:
            lo, hi = self.extrema(Y)
            phi = torch.ones_like(Y)
            for s in self.parts():
                i = self.i[s]
                r = (g[i] * taylor(self.dist[s] / (2 * self.h), self.order - 1)[:, :, None]).sum(1)
                bound = torch.where(r > 0, hi[i], lo[i])
                small = r.abs() <= 16 * 2.0 ** -52 * torch.maximum(Y[i].abs(), bound.abs())
                q = torch.clamp((bound - Y[i]) / torch.where(small, 1.0, r), min=0.0)
                v = torch.where(q > 1, (1 + 2 / q) / (1 + 1 / q + 2 / q ** 2), (q * q + 2 * q) / (q * q + q + 2))
                phi.scatter_reduce_(0, i[:, None].expand_as(v), torch.where(small, 1.0, v), "amin")
            g = g * phi[:, None, :]
        return g

    def extrema(self, Y):
        lo, hi = Y.clone(), Y.clone()
        for s in self.parts():
            i = self.i[s, None].expand(-1, Y.shape[1])
            lo.scatter_reduce_(0, i, Y[self.j[s]], "amin")
            hi.scatter_reduce_(0, i, Y[self.j[s]], "amax")
        return lo, hi

    def rhs(self, Y, orders, w=None):
        if self.kind == "weno":
            return self.rhs_weno(Y, orders)
        g = self.gradients(Y, orders)
        own, _ = self.flux(Y, w)
        total = torch.zeros_like(Y)
        for s in self.parts():
            i, j, x = self.i[s], self.j[s], self.dist[s]
            o = torch.minimum(orders[i], orders[j])
            p = taylor(x / (2 * self.h), self.order - 1)
            q = taylor(-x / (2 * self.h), self.order - 1)
            keep = torch.zeros_like(p)
            keep[:, :self.D] = (o >= 2)[:, None].to(p.dtype)
            keep[:, self.D:] = (o >= 3)[:, None].to(p.dtype)
            a = Y[i] + (g[i] * (p * keep)[:, :, None]).sum(1)
            b = Y[j] + (g[j] * (q * keep)[:, :, None]).sum(1)
            wi = None if w is None else w[i]
            (Fa, la), (Fb, lb) = self.flux(a, wi), self.flux(b, wi)
            s_max = torch.where(x > 0, 1.0, -1.0) * torch.maximum(la, lb)
            dF = 0.5 * (Fa + Fb - s_max[:, :, None] * (b - a)[:, None, :]) - own[i]
            c = self.dw[s]
            if self.order == 3:
                c = torch.where((orders[i] < 3)[:, None], self.dw_low[s], c)
            total.index_add_(0, i, (c[:, :, None] * dF).sum(1))
        return torch.where(self.bnd[:, None], 0.0, -2 * total)

    def rhs_weno(self, Y, orders):
        """Component-wise meshless WENO of local Lax-Friedrichs splittings (orders 1 and 2)."""
        F, lam = self.flux(Y)
        K = torch.zeros_like(Y)
        i, j = self.i, self.j
        for d in range(self.D):
            a = lam[:, d].clone().scatter_reduce_(0, i, lam[j, d], "amax")[:, None]
            for side, sign in ((0, 1.0), (1, -1.0)):
                if (d, side) not in self.sides:
                    mask = ((self.dist[:, d] < 0) if side == 0 else (self.dist[:, d] >= 0)).to(torch.float64)
                    self.sides[d, side] = ({q: self.slopes(q, False, mask) for q in (1, 2)}, self.sum(mask))
                one, members = self.sides[d, side]
                f = 0.5 * (F[:, d] + sign * a * Y)          # the own field; a neighbour's takes the own alpha
                df = 0.5 * (F[j, d] + sign * a[i] * Y[j]) - f[i]
                deg = torch.where((orders >= 2) & (members >= taylor(self.dist[:1], 2).shape[1]), 2, 1)
                gC = [self.sum(self.central[q][:, :, None] * df[:, None, :]) for q in (1, 2)]
                gS = [self.sum(one[q][:, :, None] * df[:, None, :]) for q in (1, 2)]
                gC = torch.where((orders >= 2)[:, None, None], gC[1], gC[0])
                gS = torch.where((deg >= 2)[:, None, None], gS[1], gS[0])
                sC, sS = (gC * gC).sum(1) * self.h ** 2, (gS * gS).sum(1) * self.h ** 2
                s2 = torch.maximum(f * f, sC)
                s2 = torch.where(s2 > 0, s2, 1.0)
                q = (sS / s2 + 1e-12) / (sC / s2 + 1e-12)
                wS = 1 / (1 + q * q)
                usable = (members >= self.D)[:, None]
                K -= torch.where(usable, wS * gS[:, d] + (1 - wS) * gC[:, d], gC[:, d])
        return torch.where(self.bnd[:, None], 0.0, K)

    # ---- one step
    def boundary(self, Y, start):
        donor = self.donor.clamp(min=0)
        src = torch.where((self.donor >= 0)[:, None], Y[donor], start)
        if self.outflow:
            kept = ~torch.isin(self.tags, torch.tensor(self.outflow, device=self.dev))
            src = torch.where(kept[:, None], start, src)
        else:
            src = start
        return torch.where(self.bnd[:, None], src, Y)

    def maxwellian(self, Y):
        u = Y.sum(1, keepdim=True)
        a = torch.tensor(BGK["macro_velocity"], dtype=torch.float64, device=self.dev)
        return (u + ((u * a)[:, None, :] * self.sinv[None]).sum(2)) / Y.shape[1]

    def implicit(self, Y, dt_ii):
        if dt_ii is None:
            return Y, (self.maxwellian(Y) - Y) / BGK["epsilon"]
        k = dt_ii / BGK["epsilon"]
        out = (Y + k * self.maxwellian(Y)) / (1 + k)
        return out, (out - Y) / dt_ii

    def step(self, U, dt):
        """One step; `dt` a number or one value per particle, (N, 1)."""
        S, orders = 3, torch.full((len(U),), self.order, device=self.dev)
        moving = self.kind == "moving"
        x0, KE, KI, KX = self.x.clone(), [], [], []
        Y = self.boundary(U.clone(), U)
        if self.Ai:
            out, ki = self.implicit(Y, None)
            KI.append(torch.where(self.bnd[:, None], 0.0, ki))
        inside = ~self.bnd
        for s in range(S):
            last = s + 1 == S
            a, ai = (self.b, self.bi) if last else (self.A[s + 1], self.Ai[s + 1] if self.Ai else None)
            w = torch.where(self.bnd[:, None], 0.0, Y[:, 1:-1] / Y[:, :1]) if moving else None
            lo, hi = self.extrema(Y)
            for _ in range(65):
                K = self.rhs(Y, orders, w)
                new = U.clone()
                for q, k in enumerate(KE + [K]):
                    new = new + dt * a[q] * k
                    if ai is not None and ai[q]:
                        new = new + dt * ai[q] * KI[q]
                ki = None
                if self.Ai and not last:
                    new, ki = self.implicit(new, dt * self.Ai[s + 1][s + 1])
                cand = Y + dt * K if self.substep else new
                pad = self.delta + self.pad * torch.maximum(lo.abs(), hi.abs())
                bad = ((hi - lo).abs() >= self.delta ** 3) & ((cand < lo - pad) | (cand > hi + pad))
                fine = torch.isfinite(cand).all(1)
                if isinstance(self.pde, package().Euler):
                    fine &= (cand[:, 0] > 0) & (cand[:, -1] - 0.5 * (cand[:, 1:-1] ** 2).sum(1) / cand[:, 0] > 0)
                drop = inside & (bad.any(1) | ~fine) & (orders > 1)
                if not bool(drop.any()):
                    break
                orders = orders - drop.long()
            KE.append(K)
            if ki is not None:
                KI.append(ki)
            Y = self.boundary(torch.where(self.bnd[:, None], U, new), U)
            if moving:
                KX.append(w)
                self.x = x0 + sum(dt * a[q] * k for q, k in enumerate(KX) if a[q])
                if not last:
                    self.dist = self.x[self.j] - self.x[self.i]
                    for d in range(self.D):
                        if self.length[d]:
                            self.dist[:, d] -= self.length[d] * torch.round(self.dist[:, d] / self.length[d])
                    self.geometry()
        if moving:
            self.search()
        return Y

    def volumes(self):
        S = 1 + self.sum(self.w)
        V = 1 / S
        V = V / S + self.sum(self.w / S[self.j] * V[self.j])
        V = V.clamp(min=0)
        return V * (math.prod(self.box) / V.sum())


def union_of(cloud):
    """The clouds of a batch side by side as one (any arrangement without neighbours across clouds)."""
    hcc, shift, pos = package(), 0.0, []
    for c in cloud:
        pos.append(c.pos - c.pos.min(axis=0) + np.array([shift, 0.0]))
        shift = pos[-1][:, 0].max() + 4 * c.radius
    cat = lambda f: np.concatenate([getattr(c, f) for c in cloud])  # noqa: E731
    pos = np.concatenate(pos)
    lo, hi = tuple(pos.min(axis=0)), tuple(pos.max(axis=0))
    c0 = cloud[0]
    return hcc.Cloud(pos, cat("is_boundary"), cat("tags"), cat("volumes"), c0.dx, c0.radius, lo, hi, lo, hi, (False, False))


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    cloud, U0, spec = make_inputs(case, seed)
    batch = case["kind"] == "bgk"
    m = Method(case, union_of(cloud) if batch else cloud, spec, dev)
    U = torch.tensor(U0, dtype=torch.float64, device=dev)
    cfl, t = cfl_of(case), 0.0
    if batch:
        of = torch.repeat_interleave(torch.arange(len(cloud), device=dev), torch.tensor([c.n for c in cloud], device=dev))
    for _ in range(case["steps"]):
        dt = m.time_step(U)
        if batch:
            dt = cfl * torch.full((len(cloud),), math.inf, dtype=torch.float64, device=dev).scatter_reduce_(0, of, dt, "amin")
            U = m.step(U, dt[of, None])
        else:
            dt = cfl * dt.min()
            U = m.step(U, dt)
        t = t + dt
    got = {"U": U.cpu().numpy(), "t": t.cpu().numpy()}
    if case["kind"] == "moving":
        got["x"], got["V"] = m.x.cpu().numpy(), m.volumes().cpu().numpy()
    return got
