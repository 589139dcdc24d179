"""Closure steps where nearly every block is dry: the kernel's groups draw many
dry blocks in a row, between the few that run the net."""
import numpy as np
import pytest

from rift_gb300 import capi, closure, synth
from test_gpu_closure_edges import SCALE, _params

pytestmark = pytest.mark.gpu

PERIOD = 256  # one pool of 21 x 30 cells in each 16 x 16 blocks


def _pools(ny, nx):
    rng = np.random.default_rng(21)
    bed, h = 10.0 + rng.uniform(0, 0.3, (PERIOD, PERIOD)), np.zeros((PERIOD, PERIOD))
    h[100:121, 75:105] = rng.uniform(0.05, 1.0, (21, 30))
    q = rng.normal(0, 0.2, (2, PERIOD, PERIOD)) * (h > 0)
    B = np.pad(np.tile(bed, (ny, nx)), ((0, 1), (0, 1)), mode="wrap")
    n = np.zeros((PERIOD * ny + 4, PERIOD * nx + 4))
    n[2:-2, 2:-2] = 0.03
    sim = capi.Sim(synth.Case(name="pools", B=B, cell=4.0, n=n, flags=synth.TILE_ACCEL)).setup()
    full = [np.pad(np.tile(a, (ny, nx)), 2) for a in (h, q[0], q[1])]
    sim.set_state(0.0, 0.1, sim.field("BC") + full[0], full[1], full[2])
    return sim


def test_long_runs_of_dry_blocks():
    """12,288 blocks, about one in 40 wet, against one pool alone: every copy
    ends bit for bit as the single one, pass after pass."""
    pytest.importorskip("torch")
    model = closure.Model(_params(np.random.default_rng(5)), SCALE, np.full(4, 2e-3, np.float32))
    sims = []
    for ny, nx in ((1, 1), (8, 6)):
        sim = _pools(ny, nx)
        run = closure.ClosureRun(sim, model, hmin=0.01, lim=0.2, tau=1e9)
        h0 = sim.field("W")
        for _ in range(5):
            run.apply(2.0, 0.0)
        closure.check(run.view.stream)
        sims.append((sim, run, h0))
    (a, ra, h0), (b, rb, _) = sims
    assert np.count_nonzero(a.field("W") != h0) > 100
    assert rb.block_counts()[0] == 48 * ra.block_counts()[0] > 0
    for f in ("W", "HU", "HV"):
        one, many = a.field(f)[2:-2, 2:-2], b.field(f)[2:-2, 2:-2]
        assert np.array_equal(many, np.tile(one, (8, 6))), f
