"""Ensemble members with fronts: water that spreads over dry land and drains
away, on grids several 60-column segments wide, so that tiles turn on and off
and are shared by the warps of the row queue.  Every member against a run of
its own, Euler members and members of two stages together."""
import numpy as np
import pytest

import fixture as FX
from rift_gb300 import capi, synth

pytestmark = pytest.mark.gpu

Q99, MAX = 1e-6, 5e-5  # the parity bars (m)

# ny, nx, Euler, tile acceleration, mounds of water (row, column, radius in cells, depth)
MEMBERS = [
    (150, 331, True, True, [(40, 60, 14, 0.5), (110, 250, 9, 0.4)]),
    (97, 410, False, True, [(30, 58, 12, 0.5), (60, 300, 12, 0.3)]),
    (211, 133, True, True, [(100, 66, 20, 0.3)]),
    (40, 90, True, False, [(20, 45, 8, 0.4)]),
    (64, 200, False, True, [(10, 119, 7, 0.6)]),
    (90, 251, True, True, []),  # dry throughout
]


def _member(api, k):
    ny, nx, euler, accel, mounds = MEMBERS[k]
    rng = np.random.default_rng(50 + k)
    X, Y = np.meshgrid(np.arange(nx + 1) * 10.0, np.arange(ny + 1) * 10.0)
    z = 50.0 - 0.004 * X - 0.002 * Y + synth.gaussian_bumps(X, Y, rng, 8, (0.2, 0.8), (60, 150), nx * 10.0)
    n = np.zeros((ny + 4, nx + 4))
    n[2:-2, 2:-2] = 0.03
    J, I = np.mgrid[0:ny, 0:nx]
    h0 = np.zeros_like(n)
    for j, i, r, d in mounds:
        h0[2:-2, 2:-2] = np.maximum(h0[2:-2, 2:-2], np.where((J - j) ** 2 + (I - i) ** 2 < r * r, d, 0.0))
    case = synth.Case(name=f"front{k}", B=z, cell=10.0, n=n, h0=h0,
                      flags=synth.H_INIT | synth.DRAIN_UNIFORM | (synth.EULER if euler else 0)
                      | (synth.TILE_ACCEL if accel else 0),
                      series={1: synth.csv_series([0, 10], [2000, 2000])})
    return capi.Sim(case, api=api).setup()


def _pair(api):
    alone = [_member(api, k) for k in range(len(MEMBERS))]
    members = [_member(api, k) for k in range(len(MEMBERS))]
    return alone, members, capi.Ensemble(members)


CALLS = (1, 1, 3, 7, 20, 40, 60, 60, 60, 60)


def test_tile_sets_follow_the_fronts(engine_api):
    alone, members, ens = _pair(engine_api)
    on, off = np.zeros(len(MEMBERS), int), np.zeros(len(MEMBERS), int)
    last = [set(s.tiles()[1]) for s in alone]
    for steps in CALLS:
        _, k = ens.run(max_steps=steps)
        assert (k == steps).all()
        for m, (a, b) in enumerate(zip(members, alone)):
            b.run(steps)
            (wa, aa), (wb, ab) = a.tiles(), b.tiles()
            assert np.array_equal(wa, wb), (m, steps, np.flatnonzero(wa != wb))
            assert np.array_equal(np.sort(aa), np.sort(ab)), (m, steps)
            d = np.abs(FX.interior(a.field("W") - b.field("W")))
            assert np.quantile(d, 0.99) <= Q99 and d.max() <= MAX, (m, steps, d.max())
            now = set(ab)
            on[m] += len(now - last[m])
            off[m] += len(last[m] - now)
            last[m] = now
    ens.close()
    assert (on[:3] >= 5).all() and (off[:3] >= 5).all(), (on, off)  # fronts advanced, tiles dried


def test_tile_speeds_and_dt_match_a_run_alone(engine_api):
    """dt is bounded by the last speeds of tiles that went inactive: a speed
    left over from an earlier step shortens it.  The speeds agree as far as the
    states do (the parity bars), t to the rounding of dt's speeds."""
    alone, members, ens = _pair(engine_api)
    for steps in CALLS:
        t, _ = ens.run(max_steps=steps)
        for m, (a, b) in enumerate(zip(members, alone)):
            tb = b.run(steps)[0]
            assert abs(t[m] - tb) <= 1e-6 * max(1.0, abs(tb)), (m, steps, t[m], tb)
            for va, vb in zip(a.tile_speeds(), b.tile_speeds()):
                assert np.allclose(va, vb, rtol=1e-3, atol=1e-4), (m, steps, np.abs(va - vb).max())
    ens.close()
