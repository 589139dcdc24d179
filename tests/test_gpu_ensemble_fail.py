"""An ensemble run whose grid barrier gives up (its poll limit set to zero): no
member goes on as if nothing had happened, and after a fresh start each one
runs as a new handle does."""
import numpy as np
import pytest

from rift_gb300 import capi, synth

pytestmark = pytest.mark.gpu


def _member(api, k):
    """A pond in dry land; member 1's is large enough for the step loop on
    listed (segment, tile row) pairs."""
    ny, nx, r = [(60, 80, 20), (560, 700, 200), (120, 150, 40)][k]
    rng = np.random.default_rng(k)
    X, Y = np.meshgrid(np.arange(nx + 1) * 10.0, np.arange(ny + 1) * 10.0)
    z = 30.0 - 0.002 * X + synth.gaussian_bumps(X, Y, rng, 6, (0.2, 0.8), (60, 150), nx * 10.0)
    n = np.zeros((ny + 4, nx + 4))
    n[2:-2, 2:-2] = 0.03
    J, I = np.mgrid[0:ny, 0:nx]
    h0 = np.zeros_like(n)
    h0[2:-2, 2:-2] = np.where((J - ny / 2) ** 2 + (I - nx / 2) ** 2 < r * r, 0.5, 0.0)
    return capi.Sim(synth.Case(name=f"pond{k}", B=z, cell=10.0, n=n, h0=h0,
                               flags=synth.H_INIT | synth.TILE_ACCEL), api=api).setup()


def test_members_of_a_failed_run_stop_and_start_again(engine_api):
    members = [_member(engine_api, k) for k in range(3)]
    ens = capi.Ensemble(members)
    ens.run(max_steps=3)
    assert 608 < members[1].tiles()[1].size < members[1].grid_size
    ens.set_wait_polls(0)
    with pytest.raises(capi.RiftError, match="timed out"):
        ens.run(max_steps=3)
    ens.set_wait_polls(-1)
    for m in members:
        with pytest.raises(capi.RiftError, match="timed out"):
            m.run(1)
    with pytest.raises(capi.RiftError, match="timed out"):
        ens.run(max_steps=1)
    for k, m in enumerate(members):
        fresh = _member(engine_api, k)
        m.init()
        for s in (m, fresh):
            s.run(30)
        assert m.time() == fresh.time()
        assert all(np.array_equal(a, b) for a, b in zip(m.tiles(), fresh.tiles()))
        assert all(np.array_equal(m.field(f), fresh.field(f)) for f in ("W", "HU", "HV"))
    ens.run(max_steps=5)
    ens.close()


def test_autotune_refuses_a_failed_member(engine_api):
    member = _member(engine_api, 0)
    ens = capi.Ensemble([member])
    ens.set_wait_polls(0)
    with pytest.raises(capi.RiftError, match="timed out"):
        ens.run(max_steps=3)
    with pytest.raises(capi.RiftError, match="timed out"):
        member.autotune(2)
    member.init()
    member.autotune(2)
    ens.close()
