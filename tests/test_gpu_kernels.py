"""Edges of the kernels' splits and tiles: sizes around a warp, a tile and a slot group, short lists and long ones,
and the options that select a branch, each against the FP64 oracle (bit for bit in FP64; FP32 within the path's stated
tolerances: right-hand sides 1e-4, states 1e-5 relative L1)."""
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RING = tuple((float(np.cos(2 * np.pi * q / 16)), float(np.sin(2 * np.pi * q / 16))) for q in range(16))
OUTFLOW = {t: 2 for t in range(1, 7)}


def _pair(hcc, oracle, cfg, cloud, U):
    g = hcc.Context(cfg)
    c64 = type(cfg)()
    for name, _ in cfg._fields_:
        setattr(c64, name, getattr(cfg, name))
    c64.precision = 0
    o = oracle.OracleContext(c64, sys.modules["hcc_gb300._abi"])
    for c in (g, o):
        c.upload_cloud(cloud)
        c.build_neighbours()
        c.prepare_geometry()
        c.upload_state(U)
    return g, o


def _rel_l1(a, b):
    return np.abs(a - b).sum() / np.abs(b).sum()


def _same_bits(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.uint64), np.ascontiguousarray(b).view(np.uint64))


def _euler(cloud, seed=0):
    rng = np.random.default_rng(seed)
    D, x = cloud.dim, cloud.pos / (np.array(cloud.domain_max) - np.array(cloud.domain_min))
    f = [1 + 0.2 * np.sin(2 * np.pi * (x @ rng.integers(1, 3, D)) + rng.uniform(0, 6)) for _ in range(D + 2)]
    u = [v - 1 for v in f[1:-1]]
    return np.column_stack([f[0]] + [f[0] * v for v in u] + [f[-1] / 0.4 + 0.5 * f[0] * sum(v * v for v in u)])


@pytest.mark.parametrize("D,n", [(1, 5), (1, 67), (2, 6), (2, 13), (3, 5), (3, 7)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_cfl_step_from_the_speed_table(hcc, oracle, cuda_lib, D, n, precision):
    """Slot counts that do and do not fill a group of four, in every dimension, stream-fed in both precisions (FP32:
    a sum of positive terms, each within a few units of round-off: 1e-5)."""
    h = 1.0 / n
    cloud = hcc.rectangular_cloud((0.0,) * D, (1.0,) * D, h, 2.5 * h, jitter=0.2 * h, seed=n)
    cfg = hcc.make_config(hcc.Euler(D), cloud, bc_map=OUTFLOW, precision=precision)
    g, o = _pair(hcc, oracle, cfg, cloud, _euler(cloud))
    g.set_tile_staging(False)
    got, want = g.time_step(), o.time_step()
    assert got == want if precision == "fp64" else abs(got - want) < 1e-5 * want


@pytest.mark.parametrize("D,cells,periodic", [(1, 9, True), (2, 6, True), (2, 4, True), (3, 4, True), (3, 6, (True, False, True)),
                                              (2, 5, (False, True)), (3, 5, False)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_geometry_of_small_boxes(hcc, oracle, cuda_lib, D, cells, periodic, precision):
    """Boxes one to three bins wide on periodic and walled axes (repeated and missing window bins), linear fits in every
    dimension, donors of every wall: lists, weights and divergence weights bit for bit, and a step's boundary states."""
    h = 0.1
    cloud = hcc.rectangular_cloud((0.0,) * D, (cells * h,) * D, h, 2.5 * h, periodic=periodic, jitter=0.2 * h, seed=3)
    pde = hcc.LinearAdvection(tuple((1.0 - 0.3 * d,) for d in range(D)))
    cfg = hcc.make_config(pde, cloud, scheme=hcc.MUSCL(2, 2), precision=precision, bc_map={1: 2, 2: 1, 3: 2, 4: 2, 5: 1, 6: 2})
    U = np.sin(5 * cloud.pos).sum(axis=1)[:, None] + 3.0
    g, o = _pair(hcc, oracle, cfg, cloud, U)
    for a, b in zip(g.neighbours(), o.neighbours()):
        assert np.array_equal(a, b) and (a.dtype != np.float64 or _same_bits(a, b))
    total = int(o.neighbour_counts().sum())
    (dg, rg, kg), (do, ro, ko) = g.geometry(total), o.geometry(total)
    assert _same_bits(dg, do) and np.array_equal(rg, ro) and np.array_equal(kg, ko)
    counts = o.neighbour_counts()[cloud.is_boundary == 0]
    assert g.counters()["min_neighbours_interior"] == counts.min()
    dt = 0.3 * o.time_step()
    g.step(0.0, dt)
    o.step(0.0, dt)
    a, b = g.download_state(), o.download_state()
    assert _same_bits(a, b) if precision == "fp64" else _rel_l1(a, b) < 1e-5


@pytest.mark.parametrize("strategy", ["EPD0", "EPD1", "EPD2"])
@pytest.mark.parametrize("criterion,flux,n", [("u1", "rusanov", 11), ("u2", "rusanov", 6), ("pad", "aligned", 9),
                                              ("only", "rusanov", 8), ("none", "aligned", 5)])
def test_wide_kinetic_passes(hcc, oracle, cuda_lib, strategy, criterion, flux, n):
    """The 16-velocity passes with lanes sharing a particle: every interface strategy and check, clouds that leave a
    partial tile."""
    h = 1.0 / n
    cloud = hcc.rectangular_cloud((0.0, 0.0), (1.0, 1.0 + h), h, 2.5 * h, jitter=0.2 * h, seed=n)
    pde = hcc.KineticRelaxation(RING, epsilon=1e-3, macro_velocity=(1.0, 0.5))
    crit = {"u1": hcc.MOODu1(1e-3), "u2": hcc.MOODu2(1e-3), "pad": hcc.MOODPAD(), "only": hcc.OnlyMOOD(),
            "none": hcc.NoMOOD()}[criterion]
    cfg = hcc.make_config(pde, cloud, scheme=hcc.MUSCL(2, 2, flux=flux), mood=hcc.MOOD(getattr(hcc, strategy), crit),
                          tableau="IMEX_ARS222", bc_map=OUTFLOW, precision="fp32")
    U = pde.maxwellian(1.0 + 0.2 * np.sin(2 * np.pi * cloud.pos[:, 0]) * np.cos(3 * cloud.pos[:, 1]))
    g, o = _pair(hcc, oracle, cfg, cloud, U.astype(np.float32).astype(np.float64))
    inner = cloud.is_boundary == 0
    assert _rel_l1(g.compute_rhs()[inner], o.compute_rhs()[inner]) < 1e-4
    dt = 0.3 * o.time_step()
    for _ in range(2):
        g.step(0.0, dt)
        o.step(0.0, dt)
    assert _rel_l1(g.download_state(), o.download_state()) < 1e-5


@pytest.mark.parametrize("D,n", [(2, 9), (2, 120), (3, 6), (3, 30)])
def test_worklists_short_and_long(hcc, oracle, cuda_lib, D, n):
    """Every particle flagged (OnlyMOOD): lists below and above the length at which a tile takes fewer warps; the orders
    and counts do not depend on round-off."""
    h = 1.0 / n
    cloud = hcc.rectangular_cloud((0.0,) * D, (1.0,) * D, h, 2.5 * h, jitter=0.2 * h, seed=n)
    cfg = hcc.make_config(hcc.Euler(D), cloud, scheme=hcc.MUSCL(2, 2), mood=hcc.MOOD(hcc.EPD1, hcc.OnlyMOOD()),
                          bc_map=OUTFLOW, precision="fp32")
    g, o = _pair(hcc, oracle, cfg, cloud, _euler(cloud).astype(np.float32).astype(np.float64))
    dt = 0.3 * o.time_step()
    g.step(0.0, dt)
    o.step(0.0, dt)
    assert np.array_equal(g.orders(), o.orders()) and np.array_equal(g.mood_flags(), o.mood_flags())
    assert _rel_l1(g.download_state(), o.download_state()) < 1e-5


@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("n", [6, 11])
def test_tile_unions(hcc, oracle, cuda_lib, n, shuffled):
    """Tile tables of a Morton-numbered cloud and of a randomly numbered one (unions of most of the cloud), partial last
    tile: the union sizes (of the interior particles' tiles, unless these are too large for two blocks an SM), and the
    tile-staged right-hand side against the oracle's."""
    h = 1.0 / n
    cloud = hcc.rectangular_cloud((0.0,) * 3, (1.0,) * 3, h, 2.5 * h, jitter=0.2 * h, seed=n)
    if shuffled:
        q = np.random.default_rng(1).permutation(cloud.n)
        cloud = hcc.Cloud(cloud.pos[q], cloud.is_boundary[q], cloud.tags[q], cloud.volumes[q], cloud.dx, cloud.radius,
                          cloud.domain_min, cloud.domain_max, cloud.canvas_min, cloud.canvas_max, cloud.periodic)
    cfg = hcc.make_config(hcc.Euler(3), cloud, scheme=hcc.MUSCL(2, 2), bc_map=OUTFLOW, precision="fp32")
    g, o = _pair(hcc, oracle, cfg, cloud, _euler(cloud).astype(np.float32).astype(np.float64))
    counts, idx, _, _ = o.neighbours()
    start = np.concatenate([[0], np.cumsum(counts)])
    inner, size = cloud.is_boundary == 0, []
    for members in (np.flatnonzero(inner), np.arange(cloud.n)):
        rows = [[idx[start[i]:start[i + 1]] for i in t if inner[i]] + [t[inner[t]]]
                for t in np.split(members, range(128, len(members), 128))]
        size.append([len(np.unique(np.concatenate(r))) for r in rows])
    got = g.tile_staging()
    if got["active"]:
        assert (got["union_entries"], got["largest_union"]) in [(sum(s), max(s)) for s in size]
        assert got["union_entries"] == sum(size[0]) or max(size[0]) > 1100       # (two blocks an SM hold 1170 to 1205)
    assert _rel_l1(g.compute_rhs()[inner], o.compute_rhs()[inner]) < 1e-4


@pytest.mark.parametrize("n", [6, 150, 160])
@pytest.mark.parametrize("kind", ["euler", "order3", "limited", "moving", "strict"])
def test_fp64_passes_on_both_sides_of_the_split(hcc, oracle, cuda_lib, kind, n):
    """FP64 clouds below and above the size up to which eight lanes share a particle, with jumps that keep the worklists
    busy: states, orders and flags bit for bit."""
    h = 1.0 / n
    cloud = hcc.rectangular_cloud((0.0, 0.0), (1.0, 1.0), h, 2.5 * h, jitter=0.2 * h, seed=n, periodic=kind == "moving")
    x, y = cloud.pos[:, 0], cloud.pos[:, 1]
    inside = (x - 0.5) ** 2 + (y - 0.45) ** 2 < 0.06
    mood = hcc.MOOD(hcc.STRICT_EPD0 if kind == "strict" else hcc.EPD1, hcc.MOODu1(1e-4 * h * h))
    bc = {} if kind == "moving" else OUTFLOW
    if kind in ("order3", "limited"):
        cfg = hcc.make_config(hcc.LinearAdvection(((1.0,), (0.5,))), cloud, mood=mood, bc_map=bc,
                              scheme=hcc.MUSCL(3, 0, "vk_hard" if kind == "limited" else "none"))
        U = (np.where(inside, 1.0, 0.0) + 0.3 * np.sin(6 * x))[:, None]
    else:
        cfg = hcc.make_config(hcc.Euler(2), cloud, mood=mood, bc_map=bc, scheme=hcc.MUSCL(2, 2))
        rho, p = np.where(inside, 1.0, 0.3), np.where(inside, 1.0, 0.2)
        U = np.column_stack([rho, 0.2 * rho, -0.1 * rho, p / 0.4 + 0.025 * rho])
    g, o = _pair(hcc, oracle, cfg, cloud, U)
    if kind == "moving":
        for c in (g, o):
            c.set_mover(hcc.mover("lagrangian"))
    dt = 0.3 * o.time_step()
    assert g.time_step() == o.time_step()
    for s in range(2):
        g.step(s * dt, dt)
        o.step(s * dt, dt)
    assert _same_bits(g.download_state(), o.download_state())
    assert np.array_equal(g.orders(), o.orders()) and np.array_equal(g.mood_flags(), o.mood_flags())
    if kind == "moving":
        assert _same_bits(g.positions(), o.positions())


@pytest.mark.parametrize("ny,on", [(63, False), (64, True)])
@pytest.mark.parametrize("kind", ["euler", "advection"])
def test_tile_staging_by_size_in_2d(hcc, oracle, cuda_lib, kind, ny, on):
    """2-D clouds on both sides of the size from which the Euler flux pass is tile-staged (scalar advection: never by
    default), partial last tile: the right-hand side against the oracle's."""
    h = 1.0 / 65
    cloud = hcc.rectangular_cloud((0.0, 0.0), (65 * h, ny * h), h, 2.5 * h, jitter=0.2 * h, seed=ny)
    if kind == "euler":
        cfg = hcc.make_config(hcc.Euler(2), cloud, scheme=hcc.MUSCL(2, 2), bc_map=OUTFLOW, precision="fp32")
        U = _euler(cloud)
    else:
        cfg = hcc.make_config(hcc.LinearAdvection(((1.0,), (0.5,))), cloud, scheme=hcc.MUSCL(2, 2), bc_map=OUTFLOW,
                              precision="fp32")
        U = (1.0 + 0.2 * np.sin(5 * cloud.pos[:, 0]) * np.cos(4 * cloud.pos[:, 1]))[:, None]
    g, o = _pair(hcc, oracle, cfg, cloud, U.astype(np.float32).astype(np.float64))
    assert bool(g.tile_staging()["active"]) == (on and kind == "euler")
    inner = cloud.is_boundary == 0
    assert _rel_l1(g.compute_rhs()[inner], o.compute_rhs()[inner]) < 1e-4


@pytest.mark.parametrize("dim,n", [(1, 37), (2, 19), (3, 9), (3, 12)])
def test_weno_lanes(hcc, oracle, cuda_lib, dim, n):
    """FP32 WENO of Euler in every dimension (3, 4 and 5 lanes a particle, partial last warps and blocks), full passes and
    worklist passes, against the oracle. The right-hand side moves by up to 7.5e-6 of its L1 norm when the state moves by
    FP32 round-off (the WENO weights are ratios), so 1e-4 holds it; states within the path's 3e-4."""
    h = 1.0 / n
    cloud = hcc.rectangular_cloud((0.0,) * dim, (1.0,) * dim, h, 2.5 * h, jitter=0.2 * h, seed=n)
    cfg = hcc.make_config(hcc.Euler(dim), cloud, scheme=hcc.WENO(2), bc_map=OUTFLOW, precision="fp32",
                          mood=hcc.MOOD(hcc.EPD1, hcc.MOODu1(1e-4 * h * h)))
    x, vel = cloud.pos, np.array([0.3, -0.2, 0.1][:dim])
    rho, p = 1.0 + 0.2 * np.prod(np.sin(2 * np.pi * x), axis=1), 1.0 + 0.1 * np.cos(2 * np.pi * x[:, 0])
    U = np.column_stack([rho] + [rho * v for v in vel] + [p / 0.4 + 0.5 * rho * (vel ** 2).sum()])
    g, o = _pair(hcc, oracle, cfg, cloud, U.astype(np.float32).astype(np.float64))
    inner = cloud.is_boundary == 0
    assert _rel_l1(g.compute_rhs()[inner], o.compute_rhs()[inner]) < 1e-4
    dt = 0.3 * o.time_step()
    for c in (g, o):
        c.step(0.0, dt)
    assert _rel_l1(g.download_state()[inner], o.download_state()[inner]) < 3e-4
