"""The persistent loop on the march's items (active sets above one tile per
CTA) against the per-tile kernels of the same engine: dense and sparse sets,
sets that change from step to step, gridded sources with tracking, outputs
and the volume ledger."""
import numpy as np
import pytest

from rift_gb300 import capi, synth

pytestmark = pytest.mark.gpu

Q99, MAX = 1e-6, 5e-5  # the parity bars (m)


def _plane(ny, nx, seed=3, cell=10.0):
    rng = np.random.default_rng(seed)
    X, Y = np.meshgrid(np.arange(nx + 1) * cell, np.arange(ny + 1) * cell)
    z = 20.0 - 0.001 * X + 0.0005 * Y + synth.gaussian_bumps(X, Y, rng, 12, (0.5, 2), (40, 200), nx * cell)
    n = np.zeros((ny + 4, nx + 4))
    n[2:-2, 2:-2] = 0.03
    return z, n


def _case(name):
    ny, nx = (431, 517) if name != "front" else (700, 640)
    z, n = _plane(ny, nx)
    case = synth.Case(name=name, B=z, cell=10.0, n=n, flags=synth.TILE_ACCEL)
    rng = np.random.default_rng(5)
    if name in ("rain", "noaccel"):
        case.flags = synth.RAIN_UNIFORM | (synth.TILE_ACCEL if name == "rain" else 0)
        case.series = {0: synth.csv_series([0, 1], [50, 50])}
    if name in ("infil", "front"):  # infiltration; front: a mound that spreads over dry land
        case.flags |= synth.INFILTRATION
        case.psi, case.dtheta = 0.11, 0.3
        case.K = np.zeros_like(n)
        case.K[2:-2, 2:-2] = 1e-6 * rng.uniform(0.5, 2.0, (ny, nx))
    if name == "infil":
        case.flags |= synth.RAIN_UNIFORM
        case.series = {0: synth.csv_series([0, 1], [50, 50])}
    if name == "front":
        J, I = np.mgrid[0:ny, 0:nx]
        case.h0 = np.zeros_like(n)
        case.h0[2:-2, 2:-2] = np.where((J - ny / 2) ** 2 + (I - nx / 2) ** 2 < 200 ** 2, 0.6, 0.0)
        case.flags |= synth.H_INIT | synth.POINT_SOURCE
        case.series = {2: synth.csv_series([0, 1, 2], [300, 400, 0])}
        case.src_idx = np.array([(ny // 2) * (nx + 4) + nx // 2], dtype=np.int32)
    if name == "friction":  # fast thin flow that a rough bed stops: the speeds fall steeply
        case.n[2:-2, 2:-2] = 0.4
        case.h0 = np.zeros_like(n)
        case.h0[2:-2, 2:-2] = rng.uniform(0.0, 0.05, (ny, nx))
        case.flags |= synth.H_INIT
    if name == "maps":
        case.flags |= (synth.RAIN_GRID | synth.DRAIN_GRID | synth.SURGE_GRID | synth.CHECK_VOLUME
                       | synth.SAVE_MAX | synth.SAVE_ARRIVAL)
    return case, (ny, nx)


def _run(api, case, shape, persist, steps):
    sim = capi.Sim(case, api=api).set_schedule(1 << 30).set_persistent(1 << 30 if persist else 0).setup()
    if case.name == "maps":  # rain on one half only: dry tiles, and tiles the maps wet again
        ny, nx = shape
        r = np.zeros((ny + 4, nx + 4))
        r[2:-2, 2:nx // 2] = 30.0 / 3.6e6
        r[2:40, nx - 60:nx - 20] = 60.0 / 3.6e6
        sim.set_map(0, r)
        sim.set_map(1, np.full_like(r, 2.0 / 3.6e6))
        s = np.full_like(r, -9999.0)
        s[2:-2, 2:6] = 0.3
        sim.set_map(2, s)
    if case.name == "friction":
        q = np.random.default_rng(6).normal(0.0, 0.05, (2, *case.n.shape)) * (case.h0 > 0.02)
        sim.run(1)  # (a first step: the loop of the next launch is chosen by its active tiles)
        sim.set_state(sim.time()[0], sim.time()[1], sim.field("W"), q[0], q[1])
    for k in steps:
        sim.run(k)
    return sim


@pytest.mark.parametrize("name", ["rain", "noaccel", "infil", "front", "maps", "friction"])
def test_flow_matches_tiles(engine_api, name):
    case, shape = _case(name)
    steps = (1, 2, 30, 7)
    a = _run(engine_api, case, shape, True, steps)
    b = _run(engine_api, case, shape, False, steps)
    n = 40 + (name == "friction")
    assert a.path_stats() == (n, 0) and b.path_stats() == (0, n)
    (wa, aa), (wb, ab) = a.tiles(), b.tiles()
    # the first steps have every tile active, and the loop changes over only
    # well below one tile per CTA (608)
    assert a.grid_size > 608 and aa.size > 456
    assert np.array_equal(wa, wb) and np.array_equal(aa, ab)
    assert abs(a.time()[0] - b.time()[0]) <= 1e-6 * max(1.0, b.time()[0])
    if name != "maps":  # one statement of the arithmetic, the dt speeds included
        assert a.time() == b.time()
        assert all(np.array_equal(a.field(f), b.field(f)) for f in ("W", "HU", "HV"))
    fields = ["W"] + (["F"] if case.K is not None else [])
    fields += ["HMAX", "TWET"] if case.flags & synth.SAVE_MAX else []
    for f in fields:
        d = np.abs(a.field(f) - b.field(f))[2:-2, 2:-2]
        q, m = (Q99, MAX) if f != "TWET" else (1e-3, 1.0)
        assert np.quantile(d, 0.99) <= q and d.max() <= m, (f, d.max())
    mxa, mya = a.tile_speeds()
    mxb, myb = b.tile_speeds()
    assert np.allclose(mxa, mxb, rtol=1e-3, atol=1e-4) and np.allclose(mya, myb, rtol=1e-3, atol=1e-4)
    if case.flags & synth.CHECK_VOLUME:
        la, lb = a.ledger(), b.ledger()
        moved = sum(abs(lb[k]) for k in ("added", "drained", "surge", "boundary"))
        assert all(abs(la[k] - lb[k]) <= 1e-4 * moved for k in lb if k != "residual"), (la, lb)


@pytest.mark.parametrize("dries", [False, True])
@pytest.mark.parametrize("n", [150, 200, 340])  # 110, 195 and 550 tiles: around one per SM, below one per CTA
def test_full_rain_grid_matches_tiles(engine_api, n, dries):
    """Runs under rain maps and a drain with every tile active (and, with dries,
    a corner whose rain stops and drains away, so that the set shrinks)."""
    z, mann = _plane(n, n)
    case = synth.Case(name="rows", B=z, cell=10.0, n=mann, series={1: synth.csv_series([0, 1], [2, 2])},
                      flags=synth.RAIN_GRID | synth.DRAIN_UNIFORM | synth.TILE_ACCEL)
    sims = []
    for persist in (1 << 30, 0):
        sim = capi.Sim(case, api=engine_api).set_schedule(1 << 30).set_persistent(persist).setup()
        r = np.zeros((n + 4, n + 4))
        r[2:-2, 2:-2] = 30.0 / 3.6e6
        sim.set_map(0, r)
        sim.run(12)
        if dries:
            r[:n // 2, :n // 2] = 0.0
            sim.set_map(0, r)
            w = np.where(r > 0, sim.field("W"), sim.field("BC"))
            sim.set_state(*sim.time(), w, sim.field("HU") * (r > 0), sim.field("HV") * (r > 0))
        for k in (1, 20, 7, 30):
            sim.run(k)
        sims.append(sim)
    a, b = sims
    assert a.path_stats() == (70, 0) and b.path_stats() == (0, 70)
    (wa, aa), (wb, ab) = a.tiles(), b.tiles()
    assert (aa.size < a.grid_size) == dries
    assert np.array_equal(wa, wb) and np.array_equal(aa, ab)
    d = np.abs(a.field("W") - b.field("W"))[2:-2, 2:-2]
    assert np.quantile(d, 0.99) <= Q99 and d.max() <= MAX
