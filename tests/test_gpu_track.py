"""Re-wet tracking of inactive tiles, a warp per tile: a single cell with rain
(held and interpolated maps) or a surge depth, anywhere in a tile and in the
ragged tiles at the far edges, wets the same tiles as in the oracle."""
import numpy as np
import pytest

from rift_gb300 import capi, synth

pytestmark = pytest.mark.gpu


def _sim(api, seed, kind, **kw):
    ny, nx = 170, 205  # ragged tiles of 2 rows and 13 columns at the far edges
    rng = np.random.default_rng(seed)
    n = np.zeros((ny + 4, nx + 4))
    n[2:-2, 2:-2] = 0.03
    flags = {"rain": synth.RAIN_GRID, "surge": synth.SURGE_GRID,
             "both": synth.RAIN_GRID | synth.SURGE_GRID}[kind]
    X = np.arange(nx + 1) * 10.0
    B = np.broadcast_to(20.0 + 0.001 * X, (ny + 1, nx + 1)).copy()
    sim = capi.Sim(synth.Case(name=kind, B=B, cell=10.0, n=n, flags=flags | synth.TILE_ACCEL), api=api,
                   **kw).setup()
    cells = [np.zeros((ny + 4, nx + 4)) for _ in range(2)]
    surge = np.full((ny + 4, nx + 4), -9999.0)
    at = np.stack([rng.integers(2, ny + 2, 40), rng.integers(2, nx + 2, 40)], 1)
    at[0], at[1], at[2] = (2, nx + 1), (ny + 1, nx + 1), (ny + 1, 2)
    for k, (j, i) in enumerate(at):
        if kind == "rain" or (kind == "both" and k % 2):
            cells[k % 3 == 0][j, i] = 20.0 / 3.6e6
        else:
            surge[j, i] = 0.4 if k % 4 else 0.0
    if kind != "surge":
        sim.set_map(0, *cells)
        sim.set_map_times(0, 0.0, 1e4)
    if kind != "rain":
        sim.set_map(2, surge)
    w = sim.field("BC")
    t = sim.grid_size
    sim.set_state(600.0, 0.5, w, np.zeros_like(w), np.zeros_like(w), wet=np.zeros(t), active=[0])
    return sim


@pytest.mark.parametrize("how", ["persistent", "graph", "ensemble"])
@pytest.mark.parametrize("kind", ["rain", "surge", "both"])
def test_tracked_tiles_match_the_oracle(engine_api, oracle_api, kind, how):
    a, b = _sim(engine_api, 4, kind), _sim(oracle_api, 4, kind, create_mode=1)
    a.set_persistent(0 if how == "graph" else 1 << 30)
    ens = capi.Ensemble([a]) if how == "ensemble" else None
    for step in range(3):
        ens.run(max_steps=1) if ens else a.run(1)
        b.step()
        (wa, aa), (wb, ab) = a.tiles(), b.tiles()
        assert 20 < ab.size < b.grid_size
        assert np.array_equal(wa, wb) and np.array_equal(np.sort(aa), np.sort(ab)), (step, aa.size, ab.size)
    if ens:
        ens.close()
