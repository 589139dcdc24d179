"""A NaN in the state stays visible: the momenta it reaches, step by step, are
those it reaches in the oracle, on every schedule."""
import numpy as np
import pytest

from rift_gb300 import capi, synth

pytestmark = pytest.mark.gpu

SCHEDULES = {"persistent": (40, 1 << 30, 1 << 30), "graph, tiles": (40, 0, 1 << 30),
             "graph, march": (40, 0, 0), "persistent, march items": (420, 1 << 30, 1 << 30),
             "ensemble": (40, 1 << 30, 1 << 30)}


def _lake(api, n, flags, what, **kw):
    mann = np.zeros((n + 4, n + 4))
    mann[2:-2, 2:-2] = 0.03
    h0 = np.zeros_like(mann)
    h0[2:-2, 2:-2] = 1.0
    case = synth.Case(name="lake", B=np.full((n + 1, n + 1), 10.0), cell=10.0, n=mann, h0=h0,
                      flags=synth.H_INIT | synth.TILE_ACCEL | flags)
    sim = capi.Sim(case, api=api, **kw).setup()
    s = [sim.field(f) for f in ("W", "HU", "HV")]
    s[0 if what == "h" else 1][20, 20] = np.nan
    return sim, s


@pytest.mark.parametrize("schedule", list(SCHEDULES))
@pytest.mark.parametrize("flags", [0, synth.EULER], ids=["rk", "euler"])
@pytest.mark.parametrize("what", ["h", "hu"])
def test_nan_reaches_what_it_reaches_in_the_oracle(engine_api, oracle_api, what, flags, schedule):
    n, persist, strips = SCHEDULES[schedule]
    a, s = _lake(engine_api, n, flags, what)
    b, _ = _lake(oracle_api, n, flags, what, create_mode=1)
    a.set_persistent(persist).set_schedule(strips)
    for sim in (a, b):
        sim.set_state(1.0, 0.1, *s)
    ens = capi.Ensemble([a]) if schedule == "ensemble" else None
    for step in range(2):
        ens.run(max_steps=1) if ens else a.run(1)
        b.step()
        assert abs(a.time()[0] - b.time()[0]) <= 1e-5 * b.time()[0]
        for f in ("HU", "HV"):
            na, nb = np.isnan(a.field(f)), np.isnan(b.field(f))
            assert nb.any() and np.array_equal(na, nb), (step, f, np.argwhere(na != nb))
    if ens:
        ens.close()
