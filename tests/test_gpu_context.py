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
