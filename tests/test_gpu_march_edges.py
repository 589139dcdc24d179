"""The column march at the edges of its 60-column segments and of its items:
against the per-tile kernels of the same engine, on grids whose last segment
holds 1, 2, 59 or 60 columns and whose rows do not divide into items."""
import numpy as np
import pytest

from rift_gb300 import capi, synth

pytestmark = pytest.mark.gpu

Q99, MAX = 1e-6, 5e-5  # the parity bars (m)


@pytest.mark.parametrize("ny,nx", [(9, 59), (29, 60), (31, 61), (44, 62), (17, 120), (57, 121), (70, 183)])
@pytest.mark.parametrize("rim", [False, True])
def test_march_matches_tiles(engine_api, ny, nx, rim):
    case = synth.small_case(nx_cells=nx, ny_cells=ny, seed=nx, h0_depth=0.2, rim=rim)
    got = []
    for sched in (0, 1 << 30):
        sim = capi.Sim(case, api=engine_api).set_schedule(sched).set_persistent(0).setup()
        sim.run(25)
        got.append((sim.tiles(), sim.time()[0], sim.field("W"), sim.field("HU"), sim.field("HV")))
        sim.close()
    (t1, c1, w1, u1, v1), (t0, c0, w0, u0, v0) = got
    assert np.array_equal(t1[0], t0[0]) and np.array_equal(t1[1], t0[1])
    assert abs(c1 - c0) <= 1e-6 * max(1.0, c0)
    for a, b, k in ((w1, w0, 1.0), (u1, u0, 10.0), (v1, v0, 10.0)):
        d = np.abs(a - b)[2:-2, 2:-2]
        assert np.quantile(d, 0.99) <= k * Q99 and d.max() <= k * MAX, (d.max(), np.quantile(d, 0.99))
