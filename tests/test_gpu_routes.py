"""Sets with inactive tiles whose options have no instantiation of their own, on
the loops and sizes they are routed to, against the per-tile kernels."""
import numpy as np
import pytest

from rift_gb300 import capi, synth

pytestmark = pytest.mark.gpu

Q99, MAX = 1e-6, 5e-5  # the parity bars (m)


def _sim(api, ny, nx, flags, radius, persist, strips):
    rng = np.random.default_rng(3)
    X, Y = np.meshgrid(np.arange(nx + 1) * 10.0, np.arange(ny + 1) * 10.0)
    z = 20.0 - 0.001 * X + 0.0005 * Y + synth.gaussian_bumps(X, Y, rng, 12, (0.5, 2), (40, 200), nx * 10.0)
    n = np.zeros((ny + 4, nx + 4))
    n[2:-2, 2:-2] = 0.03
    J, I = np.mgrid[0:ny, 0:nx]
    h0 = np.zeros_like(n)
    h0[2:-2, 2:-2] = np.where((J - ny / 2) ** 2 + (I - nx / 2) ** 2 < radius ** 2, 0.6, 0.0)
    case = synth.Case(name="pond", B=z, cell=10.0, n=n, h0=h0, psi=0.11, dtheta=0.3,
                      flags=flags | synth.H_INIT | synth.TILE_ACCEL)
    if flags & synth.INFILTRATION:
        case.K = np.where(n > 0, 1e-6, 0.0)
    sim = capi.Sim(case, api=api).set_schedule(strips)
    if persist is not None:
        sim.set_persistent(persist)
    sim.setup()
    if flags & synth.RAIN_GRID:
        sim.set_map(0, np.where(h0 > 0, 20.0 / 3.6e6, 0.0))
    return sim


OUT = synth.SAVE_MAX | synth.SAVE_ARRIVAL
# rows, columns, options, radius of the pond (cells), tiles, default route of a run of 20 steps:
# steps on the loops, steps on the graph
CASES = {
    "infiltration, k_flow": (500, 620, synth.INFILTRATION | OUT, 190, (608, 760), (20, 0)),
    "infiltration, k_persist": (620, 700, synth.INFILTRATION | OUT, 250, (900, 1300), (20, 0)),
    "rain maps, k_flow": (620, 700, synth.RAIN_GRID | OUT, 250, (900, 1300), (20, 0)),
    "rain maps, graph": (1200, 1300, synth.RAIN_GRID, 540, (4096, 6000), (0, 20)),
    "rain maps, graph, tall": (1500, 2400, synth.RAIN_GRID, 700, (6500, 9000), (0, 20)),
}


@pytest.mark.parametrize("strips", [-1, 0], ids=["", "march"])
@pytest.mark.parametrize("name", list(CASES))
def test_default_route_matches_tiles(engine_api, name, strips):
    ny, nx, flags, r, (least, most), route = CASES[name]
    a = _sim(engine_api, ny, nx, flags, r, None, strips)
    b = _sim(engine_api, ny, nx, flags, r, 0, 1 << 30)
    for sim in (a, b):
        sim.run(2)  # (the first step runs on every tile: the next call's loop is chosen by the set it leaves)
    before = a.path_stats()
    for sim in (a, b):
        sim.run(1)
        sim.run(19)
    assert tuple(np.subtract(a.path_stats(), before)) == route
    (wa, aa), (wb, ab) = a.tiles(), b.tiles()
    assert least < ab.size <= most and ab.size < b.grid_size
    assert np.array_equal(wa, wb) and np.array_equal(aa, ab)
    assert abs(a.time()[0] - b.time()[0]) <= 1e-6 * max(1.0, b.time()[0])
    fields = ["W"] + (["F"] if flags & synth.INFILTRATION else []) + (["HMAX"] if flags & synth.SAVE_MAX else [])
    for f in fields:
        d = np.abs(a.field(f) - b.field(f))[2:-2, 2:-2]
        assert np.quantile(d, 0.99) <= Q99 and d.max() <= MAX, (f, d.max())
