"""The closure kernels at the edges of their tiling: one block, a single output
cell, ragged rectangles, one block more than are in flight at once (four per
SM in inference, one per SM in training), and a correction pass over a grid
of mostly dry blocks."""
import numpy as np
import pytest

from rift_gb300 import build as eb
from rift_gb300 import capi, closure, synth

from test_gpu_closure import FWD_TOL, SCALE, _params

pytestmark = pytest.mark.gpu

# (samples, height, width) of the patches; 16 x 16 output blocks
SHAPES = [(1, 22, 22), (3, 7, 7), (5, 23, 51), (153, 22, 22), (609, 22, 21), (39, 70, 70)]


@pytest.fixture(scope="module")
def torch():
    import torch
    eb.build()
    closure.load()
    return torch


def _inputs(torch, S, H, W):
    g = torch.Generator(device="cuda").manual_seed(S * 10007 + H * 101 + W)
    x = torch.randn(S, 6, H, W, generator=g, device="cuda")
    x[:, 0] = (0.3 + 0.3 * x[:, 0]).abs()
    x[:, 1:3] *= 0.2
    ramp = 0.05 * torch.arange(W, device="cuda") - 0.03 * torch.arange(H, device="cuda")[:, None]
    x[:, 3] = 30.0 + ramp + 0.2 * x[:, 3]
    x[:, 4] = 0.05 + 0.01 * x[:, 4].clamp(-3, 3)
    x[:, 5] = 1.4e-5
    p = torch.as_tensor(_params(np.random.default_rng(8)), device="cuda")
    return x.contiguous(), p, g


@pytest.mark.parametrize("S,H,W", SHAPES)
def test_forward_edges(torch, S, H, W):
    x, p, _ = _inputs(torch, S, H, W)
    out = closure.forward(x, p, SCALE)
    ref = closure.torch_forward(x * torch.as_tensor(SCALE, device="cuda").view(1, 6, 1, 1), p)
    assert out.shape == ref.shape == (S, 4, H - 6, W - 6)
    err = (out - ref).abs().max().item() / ref.abs().max().item()
    assert err < FWD_TOL, err


def _statement(torch, x, p, tgt, w, ls):
    """Loss and gradient with BF16 operands where the kernel has them, in FP64:
    the inputs relative to each 5 x 5 window's centre bed, the three layers'
    weights, both layers' activations and both layers' gradients."""
    bf = lambda a: a.to(torch.bfloat16).to(torch.float64)
    d = lambda a: a.to(torch.float64)
    unfold, fold = torch.nn.functional.unfold, torch.nn.functional.fold
    W1, b1 = p[closure.OFF_W1:closure.OFF_B1].view(32, 160), d(p[closure.OFF_B1:closure.OFF_W2])
    W2, b2 = p[closure.OFF_W2:closure.OFF_B2].view(32, 288), d(p[closure.OFF_B2:closure.OFF_W3])
    W3, b3 = p[closure.OFF_W3:closure.OFF_B3].view(8, 32)[:4], d(p[closure.OFF_B3:closure.OFF_B3 + 4])
    S, _, H, W = x.shape
    xs = x * torch.as_tensor(SCALE, device="cuda").view(1, 6, 1, 1)
    cols = unfold(xs, 5).view(S, 6, 25, -1).transpose(1, 2)      # (S, tap, channel, cell)
    bed = d(cols[:, :, 3]) - d(cols[:, 12:13, 3])
    X = bf(cols)
    X[:, :, 3] = bed                                             # (two BF16 halves: 16 bits)
    w1 = bf(W1[:, :150])
    a1 = bf(torch.relu(w1 @ X.reshape(S, 150, -1) + b1[:, None]))
    A1 = unfold(a1.view(S, 32, H - 4, W - 4), 3).view(S, 32, 9, -1).transpose(1, 2).reshape(S, 288, -1)
    w2, w3 = bf(W2), bf(W3)
    a2 = bf(torch.relu(w2 @ A1 + b2[:, None]))
    out = w3 @ a2 + b3[:, None]
    wt, diff = d(w).view(S, 4, -1), out - d(tgt).view(S, 4, -1)
    dout = 2 * ls * wt * diff
    dz2 = bf((d(W3).T @ dout) * (a2 > 0))
    dA = (w2.T @ dz2).view(S, 9, 32, -1).transpose(1, 2).reshape(S, 288, -1)
    dz1 = bf(fold(dA, (H - 4, W - 4), 3).view(S, 32, -1) * (a1 > 0))
    X[:, :, 3] = bf(bed)
    g = torch.zeros(closure.NPARAM, device="cuda", dtype=torch.float64)
    g[closure.OFF_W1:closure.OFF_B1].view(32, 160)[:, :150] = torch.einsum("sol,skl->ok", dz1, X.reshape(S, 150, -1))
    g[closure.OFF_B1:closure.OFF_W2] = dz1.sum((0, 2))
    g[closure.OFF_W2:closure.OFF_B2] = torch.einsum("sol,skl->ok", dz2, A1).flatten()
    g[closure.OFF_B2:closure.OFF_W3] = dz2.sum((0, 2))
    g[closure.OFF_W3:closure.OFF_W3 + 128] = torch.einsum("sol,skl->ok", dout, a2).flatten()
    g[closure.OFF_B3:closure.OFF_B3 + 4] = dout.sum((0, 2))
    return ls * (wt * diff ** 2).sum(), g


@pytest.mark.parametrize("S,H,W", SHAPES)
def test_train_edges(torch, S, H, W):
    """What is left between the kernel and the statement: FP32 sums (1e-6), the
    few activations that a sum's last bit moves to the next BF16 value, the bed
    in 16 bits (1.5e-5 of its range in a block), and, where blocks meet, layer-1
    gradients rounded to BF16 before they are added instead of after: random
    2^-9 of a term, so about 2^-9 of a block of the gradient at most.  The bar
    is twice that."""
    x, p, g = _inputs(torch, S, H, W)
    shape = (S, 4, H - 6, W - 6)
    tgt = torch.randn(shape, generator=g, device="cuda")
    w = (torch.rand(shape, generator=g, device="cuda") > 0.3).float()
    w[0, :, 0, 0] = 1.0
    ls = 1.0 / tgt.numel()
    grad = torch.zeros(closure.NPARAM, device="cuda")
    loss = torch.zeros(1, device="cuda", dtype=torch.float64)
    closure.train_pass(x, p, SCALE, tgt, w, ls, grad, loss)
    lref, gref = _statement(torch, x, p, tgt, w, ls)
    assert abs(loss.item() - lref.item()) <= 2.0 ** -9 * lref.item()
    for a, b in [(closure.OFF_W1, closure.OFF_B1), (closure.OFF_B1, closure.OFF_W2),
                 (closure.OFF_W2, closure.OFF_B2), (closure.OFF_B2, closure.OFF_W3),
                 (closure.OFF_W3, closure.OFF_B3), (closure.OFF_B3, closure.NPARAM)]:
        rel = ((grad[a:b] - gref[a:b]).norm() / gref[a:b].norm()).item()
        assert rel < 2.0 ** -8, (a, rel)


def _pools(ny, nx):
    """A 64-periodic bed and depth: one pool of 21 x 30 cells in each period,
    clear of its edges, over four to nine of its sixteen 16 x 16 blocks."""
    rng = np.random.default_rng(12)
    bed, h = 10.0 + rng.uniform(0, 0.3, (64, 64)), np.zeros((64, 64))
    h[20:41, 14:44] = rng.uniform(0.05, 1.0, (21, 30))
    q = rng.normal(0, 0.2, (2, 64, 64)) * (h > 0)
    B = np.tile(bed, (ny, nx))
    B = np.pad(B, ((0, 1), (0, 1)), mode="wrap")
    n = np.zeros((64 * ny + 4, 64 * nx + 4))
    n[2:-2, 2:-2] = 0.03
    sim = capi.Sim(synth.Case(name="pools", B=B, cell=4.0, n=n, flags=synth.TILE_ACCEL)).setup()
    full = [np.pad(np.tile(a, (ny, nx)), 2) for a in (h, q[0], q[1])]
    sim.set_state(0.0, 0.1, sim.field("BC") + full[0], full[1], full[2])
    return sim


def test_apply_on_mostly_dry_blocks(torch):
    """120 copies of a pool (1920 blocks, of which more hold water than are in
    flight at once, drawn from one counter) against one alone (16 blocks):
    every copy ends bit for bit as the single one, also after a second pass."""
    model = closure.Model(_params(np.random.default_rng(5)), SCALE, np.full(4, 2e-3, np.float32))
    runs = []
    for ny, nx in ((1, 1), (10, 12)):
        sim = _pools(ny, nx)
        run = closure.ClosureRun(sim, model, hmin=0.01, lim=0.2, tau=1e9)
        h0 = sim.field("W")
        for _ in range(2):
            run.apply(2.0, 0.0)
        closure.check(run.view.stream)
        runs.append((sim, run, h0))
    (a, ra, h0), (b, rb, _) = runs
    assert np.count_nonzero(a.field("W") != h0) > 100
    assert rb.block_counts()[0] == 120 * ra.block_counts()[0] > 608
    for f in ("W", "HU", "HV"):
        one, many = a.field(f)[2:-2, 2:-2], b.field(f)[2:-2, 2:-2]
        assert np.array_equal(many, np.tile(one, (10, 12))), f
