"""The kernel a bench line's roofline names is the one that ran the timed steps."""
import numpy as np
import pytest

import bench
from rift_gb300 import capi, synth


@pytest.mark.parametrize("steps, key", [((200, 0, 0), "k_persist"), ((200, 200, 0), "k_flow"),
                                        ((200, 60, 0), "k_persist+k_flow"), ((0, 0, 200), "stages"),
                                        ((64, 64, 136), "stages")])
def test_timed_kernel(steps, key):
    got, words = bench.timed_kernel(*steps)
    assert got == key
    assert all(k in words for k in key.replace("stages", "k_march").split("+"))


@pytest.mark.gpu
@pytest.mark.parametrize("side, flow", [(160, False), (480, True)])  # 110 and 1,050 tiles, all active
def test_loops_count_their_steps(engine_api, side, flow):
    n = np.zeros((side + 4, side + 4))
    n[2:-2, 2:-2] = 0.03
    z = 5.0 + 0.01 * np.arange(side + 1.0)[:, None] + np.zeros(side + 1)
    t = np.array([0.0, 1e6], dtype=np.float32)
    case = synth.Case(name="rain", B=z, cell=10.0, n=n, flags=synth.RAIN_UNIFORM | synth.TILE_ACCEL,
                      series={0: (t, np.array([40.0, 40.0], dtype=np.float32))})
    sim = capi.Sim(case, api=engine_api).setup()
    sim.step()
    sim.run(5)
    assert sim.path_stats() == (6, 0)
    assert sim.flow_steps() == (6 if flow else 0)
