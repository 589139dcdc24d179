"""The persistent loop's tile table when claims run out of CTAs: every tile of
the launch's grid is taken (or all but one) when the front moves on, so the
event that voids the table is raised, by one CTA and by several."""
import numpy as np
import pytest

from rift_gb300 import capi, synth

pytestmark = pytest.mark.gpu

Q99, MAX = 1e-6, 5e-5  # the parity bars (m)
SMS = 152


def _drops(tiles, seed=0):
    """Single wet tiles in dry land, four tiles apart, whose water spreads:
    5 `tiles` active tiles (with tile 0, one of them), more when it does."""
    side = int(np.ceil(np.sqrt(tiles)))
    nx, ny = 16 * (4 * side + 4) - 4, 14 * (4 * side + 4) - 4  # (no tile without interior cells)
    rng = np.random.default_rng(seed)
    z = 10.0 - 0.02 * np.arange(nx + 1)[None, :] + 0.02 * rng.standard_normal((ny + 1, nx + 1))
    n = np.zeros((ny + 4, nx + 4))
    n[2:-2, 2:-2] = 0.03
    h0 = np.zeros_like(n)
    for k in range(tiles):
        j, i = 2 + 14 * (4 * (k // side) + 2), 2 + 16 * (4 * (k % side) + 2)
        h0[j + 6:j + 8, i + 6:i + 10] = 0.4 + 0.2 * rng.random()
    return synth.Case(name="drops", B=z, cell=10.0, n=n, h0=h0, flags=synth.TILE_ACCEL | synth.H_INIT)


@pytest.mark.parametrize("tiles", [30, 121])  # 151 and 606 active tiles: grids of 152 and 608 CTAs
@pytest.mark.parametrize("steps", [1, 7, 100])
def test_growth_past_the_grid(engine_api, tiles, steps):
    case = _drops(tiles)
    a = capi.Sim(case, api=engine_api).setup()
    b = capi.Sim(case, api=engine_api).set_schedule(1 << 30).set_persistent(0).setup()
    for sim in (a, b):
        sim.run(2)
    assert 0 <= SMS * (4 if tiles > 30 else 1) - a.tiles()[1].size <= 3
    done = 0
    while done < 100:
        for sim in (a, b):
            sim.run(steps)
        done += steps
        (wa, aa), (wb, ab) = a.tiles(), b.tiles()
        assert np.array_equal(wa, wb) and np.array_equal(np.sort(aa), np.sort(ab)), done
    assert aa.size > SMS * (4 if tiles > 30 else 1)
    assert abs(a.time()[0] - b.time()[0]) <= 1e-6 * max(1.0, b.time()[0])
    d = np.abs(a.field("W") - b.field("W"))[2:-2, 2:-2]
    assert np.quantile(d, 0.99) <= Q99 and d.max() <= MAX, d.max()
    if steps > 1 and tiles == 30:
        assert a.table_steps() > 0


def test_channel_flood_in_one_call(engine_api):
    """The channel flood on its full grid: the first steps run on every tile,
    the next on 151 of 152 CTAs."""
    case = synth.config2(N=2048)
    a = capi.Sim(case, api=engine_api).setup()
    b = capi.Sim(case, api=engine_api).set_schedule(1 << 30).set_persistent(0).setup()
    for sim in (a, b):
        sim.run(600)
    (wa, aa), (wb, ab) = a.tiles(), b.tiles()
    assert np.array_equal(wa, wb) and np.array_equal(np.sort(aa), np.sort(ab))
    d = np.abs(a.field("W") - b.field("W"))[2:-2, 2:-2]
    assert np.quantile(d, 0.99) <= Q99 and d.max() <= MAX, d.max()


@pytest.mark.parametrize("flags", [0, synth.SAVE_MAX | synth.SAVE_ARRIVAL, synth.INFILTRATION])
def test_thin_set_past_one_tile_per_cta(engine_api, flags):
    """Strands of water a tile apart: few tiles in many strips, which stay on the
    tile loop up to two tiles per CTA of its largest grid, then on k_flow."""
    nx, ny = 16 * 60 - 4, 14 * 46 - 4
    rng = np.random.default_rng(1)
    z = 10.0 + 0.02 * rng.standard_normal((ny + 1, nx + 1))
    n = np.zeros((ny + 4, nx + 4))
    n[2:-2, 2:-2] = 0.03
    h0 = np.zeros_like(n)
    for k in range(8):  # a column of tiles and one on either side: 1,104 active tiles in 207 strips
        i = 2 + 16 * (7 * k + 6)
        h0[2:-2, i + 7:i + 9] = 0.3
    case = synth.Case(name="strands", B=z, cell=4.0, n=n, h0=h0, psi=0.11, dtheta=0.3,
                      flags=synth.TILE_ACCEL | synth.H_INIT | flags)
    if flags & synth.INFILTRATION:
        case.K = np.where(n > 0, 1e-6, 0.0)
    a = capi.Sim(case, api=engine_api).setup()
    b = capi.Sim(case, api=engine_api).set_schedule(1 << 30).set_persistent(0).setup()
    for chunk in (2, 1, 5, 60):
        for sim in (a, b):
            sim.run(chunk)
        (wa, aa), (wb, ab) = a.tiles(), b.tiles()
        assert np.array_equal(wa, wb) and np.array_equal(np.sort(aa), np.sort(ab))
        if chunk == 2:
            assert 608 < aa.size <= 1216 and len(set(zip(aa % 60 // 7, aa // 60 // 2))) > 190
            first = a.flow_steps()
        if chunk == 5:
            assert a.flow_steps() == first
    d = np.abs(a.field("W") - b.field("W"))[2:-2, 2:-2]
    assert np.quantile(d, 0.99) <= Q99 and d.max() <= MAX, d.max()
