"""What a context reports and keeps: launch counters, and clouds given one after another."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OUTFLOW = {t: 2 for t in range(1, 7)}


def _euler(cloud):
    """A smooth state: waves in the density and the pressure, a uniform velocity."""
    x, D = cloud.pos, cloud.dim
    rho = 1.0 + 0.2 * np.prod(np.sin(2 * np.pi * x), axis=1)
    p, vel = 1.0 + 0.1 * np.cos(2 * np.pi * x[:, 0]), np.array([0.3, -0.2, 0.1][:D])
    return np.column_stack([rho] + [rho * v for v in vel] + [p / 0.4 + 0.5 * rho * (vel ** 2).sum()])


def _box(hcc, D, n):
    h = 1.0 / n
    return hcc.rectangular_cloud((0.0,) * D, (1.0,) * D, h, 2.5 * h, jitter=0.2 * h, seed=n)


def _prepare(ctx, cloud):
    ctx.upload_cloud(cloud)
    ctx.build_neighbours()
    ctx.prepare_geometry()


@pytest.mark.parametrize("kind,D,tiles,launches", [("euler", 1, False, 2), ("euler", 1, True, 2), ("euler", 2, False, 2),
                                                   ("euler", 2, True, 2), ("euler", 3, False, 2), ("euler", 3, True, 1),
                                                   ("advection", 2, True, 1), ("advection", 3, True, 1)])
def test_launches_of_a_cfl_step(hcc, cuda_lib, kind, D, tiles, launches):
    """The CFL pass is the table of speeds (Euler) and the minimum, or one tile-staged pass in 3-D."""
    cloud = _box(hcc, D, {1: 500, 2: 20, 3: 9}[D])
    pde = hcc.Euler(D) if kind == "euler" else hcc.LinearAdvection(tuple((1.0 - 0.2 * d,) for d in range(D)))
    ctx = hcc.Context(hcc.make_config(pde, cloud, scheme=hcc.MUSCL(2, 2), bc_map=OUTFLOW, precision="fp32"))
    _prepare(ctx, cloud)
    ctx.set_tile_staging(tiles)
    assert bool(ctx.tile_staging()["active"]) == tiles
    ctx.upload_state(_euler(cloud) if kind == "euler" else np.ones((cloud.n, 1)))
    before = ctx.counters()["kernel_launches_total"]
    ctx.time_step()
    after = ctx.counters()
    assert after["kernel_launches"] == launches and after["kernel_launches_total"] - before == launches


def _used():
    import torch
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


def _boxes(hcc, D, sizes, seed=0):
    """Boxes of different numbers of cells a side, one spacing (so one configuration serves all, the largest one's)."""
    h = 1.0 / max(sizes)
    return [hcc.rectangular_cloud((0.0,) * D, (n * h,) * (D - 1) + (n * h + h,), h, 2.5 * h, jitter=0.2 * h, seed=seed + k)
            for k, n in enumerate(sizes)]


def test_a_smaller_cloud_gives_memory_back(hcc, cuda_lib):
    """A context that held a cloud three times as large holds what a new context takes for the second one (to a quarter,
    and to the 2 MB that the driver rounds each of some 60 buffers to)."""
    small, big = _boxes(hcc, 3, (44, 66))
    cfg = hcc.make_config(hcc.Euler(3), big, scheme=hcc.MUSCL(2, 2), bc_map=OUTFLOW)
    one = hcc.Context(cfg)
    start = _used()
    _prepare(one, small)
    need = _used() - start
    ctx = hcc.Context(cfg)
    start = _used()
    _prepare(ctx, big)
    held = _used() - start
    _prepare(ctx, small)
    assert held > 2.5 * need and _used() - start < 1.25 * need + (128 << 20)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("kind,D,sizes", [("euler", 3, (11, 7, 13, 13)), ("euler", 2, (70, 20, 75, 75)), ("weno", 3, (9, 7, 10, 10)),
                                          ("order3", 2, (24, 13, 40, 40)), ("moving", 2, (24, 13, 40, 40))])
def test_clouds_one_after_another(hcc, cuda_lib, kind, D, sizes, precision):
    """Clouds given to one context, a smaller one, a larger one and another of the same size: steps, orders and flags are
    those of a new context, bit for bit."""
    clouds = _boxes(hcc, D, sizes)
    pde = hcc.LinearAdvection(((1.0,), (0.5,))) if kind == "order3" else hcc.Euler(D)
    scheme = hcc.WENO(2) if kind == "weno" else hcc.MUSCL(3, 0, "vk_hard") if kind == "order3" else hcc.MUSCL(2, 2)
    cfg = hcc.make_config(pde, clouds[2], scheme=scheme, mood=hcc.MOOD(hcc.EPD1, hcc.MOODu1(1e-8)), bc_map=OUTFLOW,
                          precision=precision)

    def results(ctx, cloud):
        U = (np.cos(3 * cloud.pos).sum(axis=1) + 3.0)[:, None] if kind == "order3" else _euler(cloud)
        if kind != "moving":
            U = U * np.where(cloud.pos[:, :1] > 0.4, 1.0, 0.4)           # a jump: worklists
        _prepare(ctx, cloud)
        ctx.upload_state(U)
        dt = 0.1 * ctx.time_step()
        for _ in range(2):
            ctx.step(0.0, dt)
        return [np.float64(dt), ctx.download_state(), ctx.orders(), ctx.mood_flags(), ctx.positions()]

    def context():
        ctx = hcc.Context(cfg)
        if kind == "moving":
            ctx.set_mover(hcc.mover("lagrangian"))
        return ctx

    kept = context()
    for cloud in clouds:
        for a, b in zip(results(kept, cloud), results(context(), cloud)):
            assert np.ascontiguousarray(a).tobytes() == np.ascontiguousarray(b).tobytes()


@pytest.mark.parametrize("kind", ["euler", "kinetic"])
def test_default_form_follows_the_numbering(hcc, cuda_lib, kind):
    """Tile staging by default for a cloud numbered along a curve; not for the same cloud in random order or in rows of a
    long box, whose unions are too large (more than 768 entries; more than two blocks an SM hold for 16 velocities), though a
    caller can still choose it; the steps of both forms agree bit for bit."""
    h = 1.0 / 70
    curve = hcc.rectangular_cloud((0.0, 0.0), (1.0, 1.0), h, 2.5 * h, jitter=0.2 * h, seed=1)
    ring = tuple((float(np.cos(2 * np.pi * q / 16)), float(np.sin(2 * np.pi * q / 16))) for q in range(16))
    pde = hcc.Euler(2) if kind == "euler" else hcc.KineticRelaxation(ring, epsilon=1e-3, macro_velocity=(1.0, 0.5))
    q = np.random.default_rng(1).permutation(curve.n) if kind == "euler" else \
        np.argsort(np.arange(curve.n) + np.random.default_rng(1).uniform(0, 480, curve.n))

    def numbered(q):
        return hcc.Cloud(curve.pos[q], curve.is_boundary[q], curve.tags[q], curve.volumes[q], curve.dx, curve.radius,
                         curve.domain_min, curve.domain_max, curve.canvas_min, curve.canvas_max, curve.periodic)

    for cloud, default in ((numbered(np.arange(curve.n)), True), (numbered(q), False)):
        cfg = hcc.make_config(pde, cloud, scheme=hcc.MUSCL(2, 2), bc_map=OUTFLOW, precision="fp32",
                              tableau="RK3_SSP" if kind == "euler" else "IMEX_ARS222",
                              mood=hcc.MOOD(hcc.EPD1, hcc.MOODu1(1e-8)))
        ctx = hcc.Context(cfg)
        _prepare(ctx, cloud)
        got = ctx.tile_staging()
        assert bool(got["active"]) == default
        assert (got["largest_union"] <= (768 if kind == "euler" else 556)) == default
        U = _euler(cloud) if kind == "euler" else pde.maxwellian(1.0 + 0.2 * np.sin(2 * np.pi * cloud.pos[:, 0]))
        out = []
        for tiles in (False, True):
            ctx.set_tile_staging(tiles)
            assert bool(ctx.tile_staging()["active"]) == tiles
            ctx.upload_state(U)
            dt = 0.3 * ctx.time_step()
            for _ in range(2):
                ctx.step(0.0, dt)
            out.append((ctx.download_state(), ctx.orders()))
        assert out[0][0].tobytes() == out[1][0].tobytes() and np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("waves,default", [(0.9, True), (1.15, False), (1.5, True)])
def test_default_form_in_2d_follows_the_waves(hcc, cuda_lib, waves, default):
    """2-D Euler, five tiles of 128 particles on an SM: the stream-fed pass where a second wave of tiles is nearly empty."""
    import torch
    n = round((waves * 5 * 128 * torch.cuda.get_device_properties(0).multi_processor_count) ** 0.5)
    cloud = _box(hcc, 2, n)
    ctx = hcc.Context(hcc.make_config(hcc.Euler(2), cloud, scheme=hcc.MUSCL(2, 2), bc_map=OUTFLOW, precision="fp32"))
    _prepare(ctx, cloud)
    assert bool(ctx.tile_staging()["active"]) == default
