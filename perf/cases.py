"""The work that users have this framework do, as cases that can be timed.

A case is a dict of plain values; `prepare` builds what a user's program has in
hand before the call (the simulation handle with its static fields, forcing and
state; the closure's inputs and weights), `run` is one pass through the public
entry points (rift_gb300.capi, rift_gb300.closure) and returns the whole
result, `exact` is the same result in 64 bits, stated here in plain torch
without the package's code, and `work` is what one pass cannot do without.

Every state is made from the seed alone, not by running the step: a rain film
of a few millimetres that runs down the slope at its Manning velocity, with
water standing in the hollows of the terrain (dense cases), or a channel of
flowing water in dry land (the flood cases).  Forcing is constant in time, so
that a pass late in a long sequence does the work of the first one.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from rift_gb300 import capi, closure, synth

G = 9.80665
EPS = 1.19209e-07
TW, TH = 16, 14          # the activity tiles of the scheme
T0, DT0 = 600.0, 0.05    # time and last time step of the states
RAIN_MMHR, DRAIN_MMHR, FLOOD_CFS = 40.0, 5.0, 100.0
PSI, DTHETA = 0.11, 0.3


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # one step of a small catchment per call: a 1D-2D coupled model calls
        # rift_step once per time step of its own (latency and launches)
        dict(name="step_small", kind="steps", ny=61, nx=83, cell=10.0, forcing="rain", steps=1),
        # the plain 512 x 512 uniform-rain workload of bench.py: resident in
        # L2, a few tiles per SM
        dict(name="rain_512", kind="steps", ny=512, nx=512, cell=10.0, forcing="rain", steps=32),
        # the 2048 x 2048 channel flood of bench.py: mostly dry, infiltration
        # and a point hydrograph, some hundred active tiles
        dict(name="flood_2048", kind="steps", ny=2048, nx=2048, cell=5.0, forcing="flood", steps=64),
        # a ragged catchment, all wet, rain with Green-Ampt infiltration
        dict(name="catchment_ragged", kind="steps", ny=1117, nx=1531, cell=5.0,
             forcing="rain_infil", steps=16),
        # the urban rain workload of bench.py (time-interpolated rain maps,
        # drain), on a grid a quarter of its size: larger than L2, all active
        dict(name="urban_4096", kind="steps", ny=4096, nx=4096, cell=2.0, forcing="rainmap", steps=8),
        # a coast: held rain map, a surge map along one side, check_volume
        dict(name="coast_surge", kind="steps", ny=500, nx=701, cell=10.0, forcing="surge", steps=16),
        # scenarios of uneven size stepped together, as the ensemble runs of
        # bench.py do between two closure applications (8 steps)
        dict(name="ensemble_20", kind="ensemble", members=20, side0=96, side1=480, cell=5.0, steps=8),
        # a forecast cycle: restart from a host state, a few steps, the depth,
        # infiltration and peak maps read back (what bench.py times end to end)
        dict(name="restart_1024", kind="restart", ny=1024, nx=1024, cell=5.0, steps=8),
        # the closure's net on a batch of training patches (validation)
        dict(name="net_forward", kind="forward", samples=256, H=70, W=70),
        # a training pass on such a batch: loss and every gradient
        dict(name="net_train", kind="train", samples=256, H=70, W=70),
        # the closure step on a live coarse handle of a 2048 x 2048 fine grid
        dict(name="closure_apply", kind="apply", ny=1024, nx=1024, cell=4.0),
        # the time-integrated face fluxes of a fine run on the coarse faces
        # (the training targets), once per step of the fine run
        dict(name="face_flux", kind="faceflux", ny=1024, nx=1024, cell=2.0, ratio=2),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "steps", "ensemble", "restart", "forward",
                       "train", "apply", "faceflux"])
    if kind == "steps":
        forcing = rng.choice(["rain", "rain", "flood", "rain_infil", "rainmap", "rainmap", "surge"])
        ny = _log(rng, 24, 3000)
        nx = max(24, min(3600, int(ny * rng.uniform(0.5, 1.8))))
        if forcing == "flood":
            ny, nx = max(ny, 200), max(nx, 200)
        most = max(1, min(64, 40_000_000 // (ny * nx)))
        return dict(kind=kind, ny=ny, nx=nx, cell=rng.choice([2.0, 5.0, 10.0]), forcing=forcing,
                    steps=_log(rng, 1, most))
    if kind == "ensemble":
        a = _log(rng, 40, 200)
        return dict(kind=kind, members=rng.randint(2, 20), side0=a,
                    side1=_log(rng, a, 500), cell=5.0, steps=_log(rng, 2, 16))
    if kind == "restart":
        ny = _log(rng, 100, 1400)
        return dict(kind=kind, ny=ny, nx=max(64, int(ny * rng.uniform(0.6, 1.4))), cell=5.0,
                    steps=_log(rng, 1, 12))
    if kind in ("forward", "train"):
        return dict(kind=kind, samples=_log(rng, 1, 256), H=6 + rng.choice([64, 64, 16, rng.randint(1, 90)]),
                    W=6 + rng.choice([64, 64, 16, rng.randint(1, 90)]))
    if kind == "apply":
        ny = _log(rng, 60, 1300)
        return dict(kind=kind, ny=ny, nx=max(48, int(ny * rng.uniform(0.6, 1.3))), cell=4.0)
    ratio = rng.choice([1, 2])
    ny = 2 * _log(rng, 30, 700)
    return dict(kind=kind, ny=ny, nx=2 * max(24, int(ny * rng.uniform(0.3, 0.7))), cell=2.0, ratio=ratio)


# ------------------------------------------------------------------ the inputs
def _gen(seed, k=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1009 + k)
    return g


def _spectral(ny, nx, power, g):
    """A random surface with amplitude ~ 1 / frequency^power, in [0, 1]."""
    f = torch.fft.rfft2(torch.randn(ny, nx, generator=g, device="cuda", dtype=torch.float64))
    ky = torch.fft.fftfreq(ny, device="cuda", dtype=torch.float64)
    kx = torch.fft.rfftfreq(nx, device="cuda", dtype=torch.float64)
    k = torch.sqrt(ky[:, None] ** 2 + kx[None, :] ** 2)
    k[0, 0] = 1.0
    f *= k ** -power
    f[0, 0] = 0.0
    z = torch.fft.irfft2(f, s=(ny, nx))
    z -= z.min()
    return z / z.max().clamp(min=1e-12)


def _cells(c):
    """Corner values -> the mean of each cell's four corners."""
    return 0.25 * (c[1:, 1:] + c[:-1, 1:] + c[:-1, :-1] + c[1:, :-1])


def _ring(a, fill=0.0):
    """Interior cells -> the h-grid with its ring of two ghost cells."""
    return torch.nn.functional.pad(a, (2, 2, 2, 2), value=fill)


def _state(case, seed, k=0):
    """Terrain, roughness, forcing and state of one simulation (FP64 tensors
    on the device; interior cells unless said otherwise)."""
    ny, nx, cell, forcing = case["ny"], case["nx"], case["cell"], case["forcing"]
    g = _gen(seed, k)
    rand = lambda: torch.rand(ny, nx, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
    relief = min(20.0, 0.02 * cell * math.sqrt(ny * nx))
    z = 5.0 + relief * _spectral(ny + 1, nx + 1, 1.8, g)
    s = dict(ny=ny, nx=nx, cell=cell, forcing=forcing)
    s["n"] = torch.full((ny, nx), 0.035, device="cuda", dtype=torch.float64)
    if forcing == "flood":
        # a meandering channel of constant depth in dry land, falling toward
        # +x and closed at both ends
        x = torch.arange(nx + 1, device="cuda", dtype=torch.float64)[None, :]
        y = torch.arange(ny + 1, device="cuda", dtype=torch.float64)[:, None]
        yc = 0.5 * ny + 0.15 * ny * torch.sin(2 * math.pi * x / (0.6 * nx))
        inside = ((y - yc).abs() < 2.5) & (x > 3) & (x < nx - 3)
        z = z + 10.0
        z = torch.where(inside, (11.0 - 0.0005 * cell * x).expand_as(z), z)
        wetc = inside[1:, 1:] & inside[:-1, 1:] & inside[:-1, :-1] & inside[1:, :-1]
        h = torch.where(wetc, 0.6 + 0.1 * rand(), torch.zeros((), dtype=torch.float64, device="cuda"))
        s["n"] = torch.where(wetc, 0.03, 0.08).double()
        jj = int(round(float(yc[0, 8]))) - 1
        s["src"] = (jj + 2) * (nx + 4) + 8 + 2
    else:
        if forcing == "rainmap":  # buildings: blocks of 5-20 cells, 10 m high
            zb = torch.rand(ny // 24 + 2, nx // 24 + 2, generator=g, device="cuda")
            roof = torch.zeros(z.shape, dtype=torch.bool, device="cuda")
            up = zb.repeat_interleave(24, 0).repeat_interleave(24, 1)[: ny + 1, : nx + 1]
            yy = torch.arange(ny + 1, device="cuda")[:, None] % 24
            xx = torch.arange(nx + 1, device="cuda")[None, :] % 24
            roof |= (up < 0.15) & (yy > 2) & (yy < 10 + 60 * up) & (xx > 2) & (xx < 22 - 60 * up)
            z = z + 10.0 * roof
            s["n"] = torch.where(_cells(roof.double()) > 0.5, 0.015, 0.05).double()
        zc = _cells(z)
        film = 0.002 + 0.002 * rand()
        w = 33
        level = torch.nn.functional.avg_pool2d(zc[None, None], w, 1, w // 2, count_include_pad=False)[0, 0]
        h = film + torch.clamp(level - zc - 0.02, 0.0, 0.6)
    zc = _cells(z)
    p = torch.nn.functional.pad((zc + h)[None, None], (1, 1, 1, 1), mode="replicate")[0, 0]
    gx = (p[1:-1, 2:] - p[1:-1, :-2]) / (2 * cell)
    gy = (p[2:, 1:-1] - p[:-2, 1:-1]) / (2 * cell)
    slope = torch.sqrt(gx * gx + gy * gy) + 1e-6
    v = torch.clamp(torch.clamp(h, max=0.05) ** (2.0 / 3.0) * torch.sqrt(slope) / s["n"], max=0.5)
    s.update(z=z, h=h, hu=-h * v * gx / slope, hv=-h * v * gy / slope)
    s["F"] = s["K"] = None
    if forcing in ("flood", "rain_infil"):
        s["K"] = 5.0 / 3.6e6 * torch.exp(0.8 * torch.randn(ny, nx, generator=g, device="cuda",
                                                           dtype=torch.float64))
        s["F"] = 0.002 + 0.003 * rand()
    if forcing in ("rainmap", "surge"):
        maps = [torch.clamp(20.0 + 40.0 * _spectral(ny, nx, 2.5, g), min=1.0) / 3.6e6 for _ in range(2)]
        s["maps"] = maps if forcing == "rainmap" else maps[:1]
    if forcing == "surge":
        rise = torch.full((ny, nx), -9999.0, device="cuda", dtype=torch.float64)
        rise[:, :6] = 0.5 + 0.05 * rand()[:, :6]
        s["surge"] = rise
    return s


def _faces(z):
    """Elevations of the x faces (h_ny, h_nx + 1) and y faces (h_ny + 1, h_nx)
    of the h-grid from the corners: the mean of a face's two corners, the ghost
    faces copies of the faces two further in, 0 elsewhere."""
    ny, nx = z.shape[0] - 1, z.shape[1] - 1
    BX = torch.zeros(ny + 4, nx + 5, device=z.device, dtype=z.dtype)
    BY = torch.zeros(ny + 5, nx + 4, device=z.device, dtype=z.dtype)
    BX[2:-2, 2:-2] = 0.5 * (z[1:] + z[:-1])
    BY[2:-2, 2:-2] = 0.5 * (z[:, 1:] + z[:, :-1])
    BX[2:-2, 1], BX[2:-2, 0] = BX[2:-2, 3], BX[2:-2, 2]
    BX[2:-2, -2] = BX[2:-2, -4]
    BY[1, 2:-2], BY[0, 2:-2] = BY[3, 2:-2], BY[2, 2:-2]
    BY[-2, 2:-2] = BY[-4, 2:-2]
    return BX, BY


def _wet_tiles(s):
    """Tile flags of the state: a tile with a wet (or rained-on) cell."""
    ny, nx = s["ny"], s["nx"]
    nBX, nBY = -(-(nx + 4) // TW), -(-(ny + 4) // TH)
    cell = torch.zeros(nBY * TH, nBX * TW, device="cuda", dtype=torch.bool)
    cell[:ny, :nx] = s["h"] > EPS if s["forcing"] == "flood" else True
    return cell.view(nBY, TH, nBX, TW).any(3).any(1)


def _active(wet):
    a = wet.clone()
    a[1:] |= wet[:-1]
    a[:-1] |= wet[1:]
    a[:, 1:] |= wet[:, :-1]
    a[:, :-1] |= wet[:, 1:]
    a[0, 0] = True
    return a


def _host(a):
    return _ring(a).cpu().numpy()


def _sim(s, maxima=False):
    """The handle a program keeps: static fields, forcing, state."""
    fl = synth.TILE_ACCEL
    series, maps = {}, None
    long = np.array([0.0, 1e9], dtype=np.float32)
    const = lambda r: (long, np.array([r, r], dtype=np.float32))  # noqa: E731
    if s["forcing"] in ("rain", "rain_infil"):
        fl |= synth.RAIN_UNIFORM
        series[0] = const(RAIN_MMHR)
    if s["forcing"] in ("rainmap", "surge"):
        fl |= synth.RAIN_GRID
    if s["forcing"] == "rainmap":
        fl |= synth.DRAIN_UNIFORM
        series[1] = const(DRAIN_MMHR)
        maps = [_host(m) for m in s["maps"]]
    if s["forcing"] == "flood":
        fl |= synth.POINT_SOURCE
        series[2] = const(FLOOD_CFS)
    if s["K"] is not None:
        fl |= synth.INFILTRATION
    if s["forcing"] == "surge":
        fl |= synth.SURGE_GRID | synth.CHECK_VOLUME
    if maxima:
        fl |= synth.SAVE_MAX | synth.SAVE_ARRIVAL
    c = synth.Case(name=s["forcing"], B=s["z"].cpu().numpy(), cell=s["cell"], n=_host(s["n"]),
                   K=None if s["K"] is None else _host(s["K"]), psi=PSI, dtheta=DTHETA, flags=fl,
                   series=series, src_idx=np.array([s["src"]], dtype=np.int32) if "src" in s else None,
                   rain_maps=maps, map_times=(0.0, 1e7) if maps else None)
    sim = capi.Sim(c).setup()
    if s["forcing"] == "surge":
        sim.set_map(0, _host(s["maps"][0]))
        sim.set_map(2, _host(s["surge"]))
    host = _hot(s, sim)
    sim.set_state(T0, DT0, *host[:4], wet=host[4], active=host[5])
    return sim, host


def _hot(s, sim):
    """The state as a restart file has it: FP64 surface elevation, momenta,
    infiltrated depth, tile flags and active tiles."""
    w = sim.field("BC") + _host(s["h"])
    wet = _wet_tiles(s)
    return (w, _host(s["hu"]), _host(s["hv"]), None if s["F"] is None else _host(s["F"]),
            wet.cpu().numpy().astype(np.uint8).ravel(),
            torch.nonzero(_active(wet).ravel()).ravel().cpu().numpy().astype(np.int32))


class _Plane:
    """A plane of the handle's device view, for torch; it keeps the handle."""

    def __init__(self, sim, ptr, v):
        self.sim = sim
        self.__cuda_array_interface__ = {"shape": (v.rows, v.pitch), "typestr": "<f4",
                                         "data": (int(ptr), False), "version": 3, "strides": None}


def _planes(sim):
    """The interior of h, hu, hv of the handle's state (no copy)."""
    v = sim.device_view()
    return [torch.as_tensor(_Plane(sim, p, v), device="cuda")[2:v.h_ny - 2, 2:v.h_nx - 2]
            for p in (v.h, v.hu, v.hv)]


def _members(case, seed):
    rng = np.random.default_rng(case["members"])  # the sides are the case's, the fields the seed's
    out = []
    for m in range(case["members"]):
        side = [int(x) for x in rng.integers(case["side0"], case["side1"] + 1, 2)]
        out.append(_state(dict(ny=side[0], nx=side[1], cell=case["cell"], forcing="rain"), seed, m + 1))
    return out


def _patches(case, seed):
    """Patches as the training data has them: (h, hu, hv, bed, n, rain)."""
    S, H, W = case["samples"], case["H"], case["W"]
    g = _gen(seed)
    rn = lambda: torch.randn(S, 1, H, W, generator=g, device="cuda")  # noqa: E731
    blur = lambda a, k: torch.nn.functional.avg_pool2d(a, k, 1, k // 2, count_include_pad=False)  # noqa: E731
    h = torch.clamp(0.08 * blur(rn(), 5) + 0.01, min=0.0)
    hu, hv = h * (0.3 * blur(rn(), 3)), h * (0.3 * blur(rn(), 3))
    bed = 15.0 + 2.0 * blur(rn(), 9) + 0.02 * rn()
    n = 0.03 + 0.05 * (blur(rn(), 7) > 0).float()
    rain = torch.full_like(h, RAIN_MMHR / 3.6e6)
    feats = torch.cat([h, hu, hv, bed, n, rain], 1).contiguous()
    scale = np.array([30.0, 200.0, 200.0, 1.0, 20.0, closure.RAIN_SCALE], dtype=np.float32)
    tgt = torch.randn(S, 4, H - 6, W - 6, generator=g, device="cuda")
    wt = (h[:, :, 3:-3, 3:-3] > 0.01).float().expand(-1, 4, -1, -1).contiguous()
    return feats, scale, tgt, wt


def _params(seed):
    """Weights of the size training ends with, in the C layout."""
    return closure.init_params(int(seed) % (1 << 31))


# the closure's constants on a coarse run: corrections of about a tenth of the
# film's flux, applied over eight steps
CL = dict(hmin=0.01, lim=0.2, tau=0.5, dtw=1.6)
OSC = (2e-3, 4e-3, 2e-3, 4e-3)
CL_SCALE = np.array([3.0, 20.0, 20.0, 1.0, 20.0, closure.RAIN_SCALE], dtype=np.float32)


def _basin(case, seed):
    """A coarse run in flood: wide shallow water, dry high ground."""
    s = _state(dict(case, forcing="rain"), seed)
    zc = _cells(s["z"])
    level = torch.quantile(zc.ravel()[:: max(1, zc.numel() // 100_000)], 0.6)
    s["h"] = torch.clamp(level + 0.3 - zc, 0.0, 2.0)
    k = 0.2 * s["h"] / torch.clamp(s["hu"].abs() + s["hv"].abs(), min=1e-6)
    s["hu"], s["hv"] = s["hu"] * torch.clamp(k, max=1.0), s["hv"] * torch.clamp(k, max=1.0)
    dry = s["h"] <= EPS
    s["hu"][dry] = 0.0
    s["hv"][dry] = 0.0
    return s


def prepare(case, seed):
    kind = case["kind"]
    if kind == "steps":
        sim, _ = _sim(_state(case, seed))
        return dict(case=case, sim=sim, out=_planes(sim))
    if kind == "restart":
        s = _state(dict(case, forcing="rain_infil"), seed)
        sim, host = _sim(s, maxima=True)
        return dict(case=case, sim=sim, host=host)
    if kind == "ensemble":
        sims = [_sim(s)[0] for s in _members(case, seed)]
        return dict(case=case, sims=sims, ens=capi.Ensemble(sims), out=[_planes(s) for s in sims])
    if kind in ("forward", "train"):
        feats, scale, tgt, wt = _patches(case, seed)
        p = torch.as_tensor(_params(seed), device="cuda")
        return dict(case=case, feats=feats, scale=scale, tgt=tgt, wt=wt, p=p, grad=torch.zeros_like(p),
                    loss=torch.zeros(1, device="cuda", dtype=torch.float64))
    if kind == "apply":
        sim, _ = _sim(_basin(case, seed))
        model = closure.Model(_params(seed), CL_SCALE, np.array(OSC, dtype=np.float32))
        cl = closure.ClosureRun(sim, model, hmin=CL["hmin"], lim=CL["lim"], tau=CL["tau"])
        return dict(case=case, sim=sim, cl=cl, out=_planes(sim))
    sim, _ = _sim(_state(dict(case, forcing="rain"), seed))
    v = sim.device_view()
    r = case["ratio"]
    any_, anx = case["ny"] // r + 4, case["nx"] // r + 4
    acc = torch.zeros(4, any_, (anx + 31) // 32 * 32, device="cuda")
    torch.cuda.synchronize()
    return dict(case=case, sim=sim, view=v, acc=acc, anx=anx, any=any_)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "steps":
        if case["steps"] == 1:
            t, dt = state["sim"].step()
        else:
            t, dt, _ = state["sim"].run(case["steps"])
        return [*state["out"], t, dt]
    if kind == "restart":
        w, hu, hv, F, wet, act = state["host"]
        state["sim"].set_state(T0, DT0, w, hu, hv, F, wet, act)
        t, dt, _ = state["sim"].run(case["steps"])
        return [state["sim"].field(n) for n in ("H", "F", "HMAX")] + [t, dt]
    if kind == "ensemble":
        t, k = state["ens"].run(max_steps=case["steps"])
        return [p for m in state["out"] for p in m] + [t, k]
    if kind == "forward":
        return closure.forward(state["feats"], state["p"], state["scale"])
    if kind == "train":
        state["grad"].zero_()
        state["loss"].zero_()
        closure.train_pass(state["feats"], state["p"], state["scale"], state["tgt"], state["wt"],
                           1.0 / (case["samples"] * 64 * 64), state["grad"], state["loss"])
        return [state["grad"], state["loss"]]
    if kind == "apply":
        state["cl"].apply(CL["dtw"], T0)
        return [*state["out"], state["cl"].corr[:, 2:case["ny"] + 2, 2:case["nx"] + 2], state["cl"].fell]
    closure.face_flux(state["view"], case["ratio"], 0.25, state["acc"], state["anx"], state["any"])
    return state["acc"][:, 2:-2, 2:state["anx"] - 2]


# --------------------------------------------------------------- 64-bit values
def _slope(dp, dm):
    return 0.5 * torch.minimum(torch.minimum(1.3 * dp.abs(), 0.5 * (dp + dm).abs()), 1.3 * dm.abs())


def _construct(U, eM, eP, ax):
    """Face values of the cells 1 .. n-2 along `ax`: (h, hu, hv) on their plus
    and minus faces."""
    n = U[0].shape[ax]
    at = lambda a, k: a.narrow(ax, k, n - 2)  # noqa: E731  (k: 0 minus, 1 own, 2 plus)
    h = U[0]
    dP, dM = at(eP, 1) - at(eM, 2), at(eP, 0) - at(eM, 1)
    sw = _slope(dP + (at(h, 2) - at(h, 1)), dM + (at(h, 1) - at(h, 0)))
    hP, hM = at(h, 1) + sw - at(eP, 1), at(h, 1) - sw - at(eM, 1)
    bar = 2 * at(h, 1) - (at(eP, 1) + at(eM, 1))
    neg = hP < 0
    hM, hP = torch.where(neg, bar, hM), torch.where(neg, 0.0, hP)
    neg = hM < 0
    hP, hM = torch.where(neg, bar, hP), torch.where(neg, 0.0, hM)
    P, M = [hP], [hM]
    for q in U[1:]:
        s = _slope(at(q, 2) - at(q, 1), at(q, 1) - at(q, 0))
        P.append(at(q, 1) + s)
        M.append(at(q, 1) - s)
    return P, M


def _factor(h, kappa):
    return 2 * h / (h * h + torch.clamp(h * h, min=kappa))


def _flux(L, R, kappa, ax):
    """Central-upwind flux and local speed from the face values left and right."""
    side = []
    for h, qu, qv in (L, R):
        r = _factor(h, kappa)
        u, v = qu * r, qv * r
        c = torch.sqrt(G * torch.clamp(h, min=0.0))
        a = u if ax == 1 else v
        inf = torch.full_like(h, math.inf)
        hi, lo = torch.where(h >= 0, a + c, -inf), torch.where(h >= 0, a - c, inf)
        f = [h * a, h * u * a, h * v * a]
        f[1 if ax == 1 else 2] = f[1 if ax == 1 else 2] + 0.5 * G * h * h
        side.append((h, h * u, h * v, hi, lo, [torch.where(h > 0, x, 0.0) for x in f]))
    (hL, uL, vL, hiL, loL, fL), (hR, uR, vR, hiR, loR, fR) = side
    ap = torch.clamp(torch.maximum(hiL, hiR), min=0.0)
    am = torch.clamp(torch.minimum(loL, loR), max=0.0)
    d = ap - am
    r = torch.where(d > 0, 1.0 / torch.where(d > 0, d, 1.0), 0.0)
    k = ap * am * r
    return ([(ap * a - am * b) * r + k * e for a, b, e in zip(fL, fR, (hR - hL, uR - uL, vR - vL))],
            torch.maximum(ap, -am))


def _face_fluxes(U, E, kappa):
    """Fluxes through the x faces (ny, nx + 1) and y faces (ny + 1, nx) of the
    interior, and the local speeds there."""
    rows, cols = slice(2, -2), slice(2, -2)
    P, M = _construct([q[rows] for q in U], E[0][rows], E[1][rows], 1)
    fx, sx = _flux([p[:, :-1] for p in P], [m[:, 1:] for m in M], kappa, 1)
    P, M = _construct([q[:, cols] for q in U], E[2][:, cols], E[3][:, cols], 0)
    fy, sy = _flux([p[:-1] for p in P], [m[1:] for m in M], kappa, 0)
    return fx, sx, fy, sy


def _ghosts(U):
    """Critical-depth outflow in the ghost ring, in place."""
    h, hu, hv = U
    crit = lambda q, d: torch.minimum((q * q / G) ** (1.0 / 3.0), d)  # noqa: E731
    for c, gs in ((2, (0, 1)), (-3, (-2, -1))):
        d = crit(hu[2:-2, c], h[2:-2, c])
        d = torch.where(d > EPS, d, 0.0)
        e = crit(hv[c, 2:-2], h[c, 2:-2])
        for k in gs:
            h[2:-2, k], hu[2:-2, k], hv[2:-2, k] = d, hu[2:-2, c], hv[2:-2, c]
            h[k, 2:-2], hu[k, 2:-2], hv[k, 2:-2] = e, hu[c, 2:-2], hv[c, 2:-2]


def _offsets(s):
    """Face elevations relative to each cell's reference elevation (a ghost
    cell takes that of the interior cell it copies)."""
    BX, BY = _faces(s["z"])
    BC = 0.25 * (BX[:, 1:] + BX[:, :-1] + BY[1:] + BY[:-1])
    BC[:2], BC[:, :2] = 0.0, 0.0
    ref = BC.clone()
    ref[2:-2, :2], ref[2:-2, -2:] = BC[2:-2, 2:3], BC[2:-2, -3:-2]
    ref[:2, 2:-2], ref[-2:, 2:-2] = BC[2:3, 2:-2], BC[-3:-2, 2:-2]
    return [BX[:, :-1] - ref, BX[:, 1:] - ref, BY[:-1] - ref, BY[1:] - ref]


def _kappa(cell):
    return math.sqrt(0.01 * max(1.0, cell))


def _steps64(s, steps):
    """`steps` steps of the scheme; h, hu, hv of the interior, t, dt, F, peak depth."""
    ny, nx, dx = s["ny"], s["nx"], s["cell"]
    kappa = _kappa(dx)
    E = _offsets(s)
    U = [_ring(s[q]) for q in ("h", "hu", "hv")]
    _ghosts(U)
    I = (slice(2, -2), slice(2, -2))
    sx_, sy_ = E[1][I] - E[0][I], E[3][I] - E[2][I]
    wet = _wet_tiles(s)
    nBY, nBX = wet.shape
    mx = torch.zeros(nBY, nBX, device="cuda", dtype=torch.float64)
    my = mx.clone()
    tiles = lambda a: torch.nn.functional.pad(  # noqa: E731
        a.double(), (0, nBX * TW - nx, 0, nBY * TH - ny)).view(nBY, TH, nBX, TW).amax((1, 3))
    has = tiles(torch.ones(ny, nx, device="cuda")) > 0
    cells = lambda a: a.repeat_interleave(TH, 0).repeat_interleave(TW, 1)[:ny, :nx]  # noqa: E731
    uniform = RAIN_MMHR / 3.6e6 if s["forcing"] in ("rain", "rain_infil") else 0.0
    drain = DRAIN_MMHR / 3.6e6 if s["forcing"] == "rainmap" else 0.0
    t, dt_prev, F = T0, DT0, s["F"]
    hmax = torch.zeros(ny, nx, device="cuda", dtype=torch.float64)
    src = None
    if "src" in s:
        src = divmod(s["src"], nx + 4)
        src = (src[0] - 2, src[1] - 2, FLOOD_CFS / 35.3147 / dx / dx)

    def flux(V, on):
        fx, vx, fy, vy = _face_fluxes(V, E, kappa)
        div = [-(a[:, 1:] - a[:, :-1]) / dx - (b[1:] - b[:-1]) / dx for a, b in zip(fx, fy)]
        hC = V[0][I]
        div[1] = div[1] - G * hC * sx_ / dx
        div[2] = div[2] - G * hC * sy_ / dx
        seen = on & has
        mx.copy_(torch.where(seen, tiles(vx[:, 1:]), mx))
        my.copy_(torch.where(seen, tiles(vy[1:]), my))
        return div

    def sources(div, hC, dt, Fc):
        S = uniform + rain
        if drain:
            S = S - torch.clamp(hC / dt, max=drain)
        if src:
            S = S + torch.zeros_like(hC).index_put_((torch.tensor(src[0], device="cuda"),
                                                     torch.tensor(src[1], device="cuda")),
                                                    torch.tensor(src[2], device="cuda", dtype=torch.float64))
        dF = None
        if Fc is not None:
            K = s["K"]
            p1, p2 = K * dt - 2 * Fc, K * (Fc + PSI * DTHETA)
            root = torch.sqrt(p1 * p1 + 8 * p2 * dt)
            dF = torch.where(p1 >= 0, (p1 + root) / (2 * dt), 4 * p2 / (root - p1))
            dF = torch.clamp(torch.minimum(dF, hC / dt), min=0.0)
            S = S - dF
        return div[0] + S, dF

    for _ in range(steps):
        on = _active(wet)
        act = cells(on)
        rain = torch.zeros((), device="cuda", dtype=torch.float64)
        if "maps" in s:
            m = s["maps"]
            rain = m[0] if len(m) == 1 else (t / 1e7) * (m[1] - m[0]) + m[0]
        div = flux(U, on)
        top = [max(float(v.max()) / 0.25, kappa) for v in (mx, my)]
        dt = min(dx / top[0], dx / top[1])
        t += dt
        h, hu, hv = (q[I] for q in U)
        hc = torch.where(h > EPS, h, 0.0)
        dh, dF = sources(div, h, dt_prev, F)
        if "surge" in s:
            up = s["surge"]
            dh = torch.where(up > 0, (up - (hc + dh * dt)) / dt, dh)
        den = h * h + torch.clamp(h * h, min=kappa)
        fric = -4 * G * s["n"] ** 2 * torch.sqrt(hu * hu + hv * hv) * h ** (5.0 / 3.0) / den ** 2
        new = [hc + dh * dt, (hu + div[1] * dt) / (1 - dt * fric), (hv + div[2] * dt) / (1 - dt * fric)]
        new[0] = torch.where(new[0] > EPS, new[0], 0.0)
        V = [q.clone() for q in U]
        for v, x, o in zip(V, new, U):
            v[I] = torch.where(act, x, o[I])
        _ghosts(V)
        F1 = None if F is None else torch.where(act, F + dF * dt, F)
        div = flux(V, on)
        h1, hu1, hv1 = (q[I] for q in V)
        dh, dF = sources(div, h1, dt, F1)
        new = [0.5 * (hc + torch.where(h1 > EPS, h1, 0.0) + dh * dt), 0.5 * (hu + hu1 + div[1] * dt),
               0.5 * (hv + hv1 + div[2] * dt)]
        new[0] = torch.where(new[0] > EPS, new[0], 0.0)
        W = [q.clone() for q in U]
        for v, x, o in zip(W, new, U):
            v[I] = torch.where(act, x, o[I])
        _ghosts(W)
        if F is not None:
            F = torch.where(act, 0.5 * (F + F1 + dF * dt), F)
        hmax = torch.maximum(hmax, torch.where(act, new[0], 0.0))
        hit = W[0][I] > EPS if not (uniform or "maps" in s) else torch.ones_like(act)
        if src:
            hit[src[0], src[1]] = True
        wet = torch.where(on & has, tiles(hit) > 0, wet)
        U, dt_prev = W, dt
    return [q[I].clone() for q in U], t, dt_prev, F, hmax


def _net64(x, p):
    """The closure's net on scaled inputs (S, 6, H, W), 64 bits."""
    F = torch.nn.functional
    W1 = p[:5120].view(32, 160)[:, :150].view(32, 5, 5, 6).permute(0, 3, 1, 2)
    W2 = p[5152:14368].view(32, 3, 3, 32).permute(0, 3, 1, 2)
    W3 = p[14400:14656].view(8, 32)[:4].view(4, 32, 1, 1)
    b1, b2, b3 = p[5120:5152], p[14368:14400], p[14656:14660]
    z1 = F.conv2d(x, W1) - x[:, 3:4, 2:-2, 2:-2] * W1[:, 3].sum(dim=(1, 2)).view(1, -1, 1, 1)
    a1 = torch.relu(z1 + b1.view(1, -1, 1, 1))
    a2 = torch.relu(F.conv2d(a1, W2) + b2.view(1, -1, 1, 1))
    return F.conv2d(a2, W3) + b3.view(1, -1, 1, 1)


def _apply64(case, seed):
    s = _basin(case, seed)
    ny, nx, cell, dtw = s["ny"], s["nx"], s["cell"], CL["dtw"]
    rep = lambda a, k: torch.nn.functional.pad(a[None, None], (k, k, k, k), mode="replicate")[0, 0]  # noqa: E731
    # the net sees the handle's ring of two ghost cells, its edge repeated
    U = [_ring(s[q]) for q in ("h", "hu", "hv")]
    _ghosts(U)
    planes = [rep(q, 1) for q in U] + [rep(_cells(s["z"]), 3), rep(s["n"], 3)]
    planes.append(torch.full_like(planes[0], float(np.float32(RAIN_MMHR)) / 3.6e6))
    x = torch.stack([q * float(c) for q, c in zip(planes, CL_SCALE)])[None]
    p = torch.as_tensor(_params(seed), device="cuda").double()
    o = _net64(x, p)[0]
    h = s["h"]
    corr = torch.zeros(4, ny, nx, device="cuda", dtype=torch.float64)
    ind = torch.zeros(ny, nx, device="cuda", dtype=torch.float64)
    for f in range(2):
        d = 1 - f  # the dimension along which the neighbour lies
        hn = torch.roll(h, -1, d)
        ok = (h > CL["hmin"]) & (hn > CL["hmin"])
        ok[0], ok[-1], ok[:, 0], ok[:, -1] = False, False, False, False
        ok.select(d, -2).fill_(False)
        m = torch.where(ok, o[2 * f] * OSC[2 * f], 0.0)
        hd = torch.where(ok, torch.where(m > 0, h, hn), 1.0)
        ind = torch.maximum(ind, m.abs() * dtw / cell / hd)
        cap = CL["lim"] * hd * cell / dtw
        corr[2 * f] = torch.maximum(torch.minimum(m, cap), -cap)
        corr[2 * f + 1] = torch.where(ok, o[2 * f + 1] * OSC[2 * f + 1], 0.0)
    by, bx = -(-ny // 16), -(-nx // 16)
    pad = torch.nn.functional.pad(ind, (0, bx * 16 - nx, 0, by * 16 - ny))
    fell = pad.view(by, 16, bx, 16).amax((1, 3)) > CL["tau"]
    own = fell.repeat_interleave(16, 0).repeat_interleave(16, 1)[:ny, :nx]
    corr[:, own] = 0.0
    c = corr.clone()
    for f in range(2):
        d = 1 - f
        other = torch.roll(own, -1, d)
        other.select(d, -1).fill_(False)
        c[2 * f: 2 * f + 2, other] = 0.0
    sh = lambda a, d: a - torch.nn.functional.pad(a, (1, 0) if d == 1 else (0, 0, 1, 0))[  # noqa: E731
        (slice(None), slice(0, -1)) if d == 1 else (slice(0, -1), slice(None))]
    k = dtw / cell
    return [h - k * sh(c[0], 1) - k * sh(c[2], 0), s["hu"] - k * sh(c[1], 1), s["hv"] - k * sh(c[3], 0),
            corr, None]


def exact(case, seed):
    kind = case["kind"]
    if kind == "steps":
        U, t, dt, _, _ = _steps64(_state(case, seed), case["steps"])
        return [*U, t, dt]
    if kind == "restart":
        U, t, dt, F, hmax = _steps64(_state(dict(case, forcing="rain_infil"), seed), case["steps"])
        return [_ring(U[0]), _ring(F), _ring(hmax), t, dt]
    if kind == "ensemble":
        got = [_steps64(s, case["steps"]) for s in _members(case, seed)]
        return [q for r in got for q in r[0]] + [np.array([r[1] for r in got]), None]
    if kind in ("forward", "train"):
        feats, scale, tgt, wt = _patches(case, seed)
        x = feats.double() * torch.as_tensor(scale, device="cuda").double().view(1, 6, 1, 1)
        p = torch.as_tensor(_params(seed), device="cuda").double()
        if kind == "forward":
            return _net64(x, p)
        grad, loss = torch.zeros_like(p), torch.zeros(1, device="cuda", dtype=torch.float64)
        for k in range(0, len(x), 16):
            q = p.clone().requires_grad_(True)
            d = _net64(x[k:k + 16], q) - tgt[k:k + 16].double()
            e = (wt[k:k + 16].double() * d * d).sum() / (case["samples"] * 64 * 64)
            e.backward()
            grad += q.grad
            loss += e.detach()
        return [grad, loss]
    if kind == "apply":
        return _apply64(case, seed)
    s = _state(dict(case, forcing="rain"), seed)
    U = [_ring(s[q]) for q in ("h", "hu", "hv")]
    _ghosts(U)
    fx, _, fy, _ = _face_fluxes(U, _offsets(s), _kappa(s["cell"]))
    e, n = [f[:, 1:] for f in (fx[0], fx[1])], [f[1:] for f in (fy[0], fy[2])]
    if case["ratio"] == 2:
        e = [0.5 * (f[0::2, 1::2] + f[1::2, 1::2]) for f in e]
        n = [0.5 * (f[1::2, 0::2] + f[1::2, 1::2]) for f in n]
    return 0.25 * torch.stack(e + n)


# ------------------------------------------------------------- the least work
# Per active cell and step: h, hu, hv read and written, the four face offsets
# and n read (a step's dt needs the whole grid, so steps cannot share a read of
# a grid larger than the caches); infiltration adds K and F, a map its planes.
# Two flux evaluations of about 170 operations per cell each, and the updates.
WORDS = dict(rain=11, rain_infil=14, flood=14, rainmap=13, surge=13)
OPS = 400
NET_FLOPS = 2 * (6 * 32 * 25 + 32 * 32 * 9 + 32 * 4)


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        a, b = case["side0"], case["side1"]
        cells = case["members"] * (0.5 * (a + b)) ** 2 * case["steps"]
        return dict(bytes=cells * 44, flops=cells * OPS)
    if kind in ("forward", "train"):
        S, H, W = case["samples"], case["H"], case["W"]
        out = S * (H - 6) * (W - 6)
        if kind == "forward":
            return dict(bytes=4 * (S * 6 * H * W + 4 * out), flops=out * NET_FLOPS)
        return dict(bytes=4 * (S * 6 * H * W + 8 * out + 2 * 14664),
                    flops=out * (3 * NET_FLOPS - 2 * 6 * 32 * 25))
    cells = case["ny"] * case["nx"]
    if kind == "apply":  # about two thirds of the cells lie under water
        return dict(bytes=cells * 4 * (5 + 4 + 3), flops=0.67 * cells * NET_FLOPS)
    if kind == "faceflux":
        return dict(bytes=4 * (7 * cells + 8 * cells / case["ratio"] ** 2), flops=130 * cells)
    if kind == "restart":  # FP64 host arrays in and out, and the steps
        return dict(bytes=cells * (4 * 8 + 3 * 8 + 4 * 7 + case["steps"] * 4 * (14 + 3)),
                    flops=cells * OPS * case["steps"])
    if case["forcing"] == "flood":  # the channel and the tiles beside it
        cells = 1.3 * case["nx"] * 3 * TH
    return dict(bytes=cells * 4 * WORDS[case["forcing"]] * case["steps"], flops=cells * OPS * case["steps"])
