"""The tile convolutions (8 x 16-pixel tiles from swizzled tensor copies) at
the sizes where they can go wrong, against the FP64 oracle on the same BF16
values: one pixel past and short of a tile, single rows, odd low-resolution
sizes, 16- and 32-channel slabs, resident and streamed weights, several
output-channel tiles, rings that wrap.  Tolerance: FP32 accumulation of at
most 9 x 288 products, |err| <= K 2^-24 sum |x w| in the worst case; 1e-4
relative (1e-5 of the largest value for sums that cancel) is above it for
these inputs and far below any indexing mistake.  Gradients in BF16 add one
rounding (2^-8)."""
import numpy as np
import pytest

from oracle import unet_oracle as U

pytestmark = pytest.mark.gpu

CASES = [  # N, H, W, C1, up1, C2, Cout
    (1, 1, 64, 32, 0, 0, 16),      # one row, the narrowest row-order width
    (1, 17, 65, 32, 0, 0, 32),     # one pixel past a tile both ways
    (2, 15, 71, 16, 0, 0, 32),     # 16-channel slabs, one pixel short
    (1, 16, 72, 48, 0, 16, 48),    # two full-resolution sources, 16-channel slabs
    (1, 33, 80, 64, 0, 32, 96),    # two sources, 32-channel slabs
    (1, 33, 64, 128, 0, 0, 160),   # streamed weights: two tiles per unit, two output tiles
    (1, 20, 66, 96, 0, 0, 256),    # four output tiles of streamed weights
    (1, 34, 66, 64, 1, 32, 32),    # upsampled + skip, odd low-resolution size
    (1, 18, 80, 32, 1, 0, 64),     # upsampled source alone
    (2, 32, 64, 96, 1, 64, 64),    # upsampled + skip, streamed weights
    (1, 18, 68, 160, 1, 128, 128),  # 288 inputs: two output tiles of four accumulators
    (1, 20, 70, 48, 1, 16, 16),    # upsampled + skip, 16-channel slabs
    (6, 48, 128, 32, 0, 0, 32),    # several tiles per CTA: rings and accumulators wrap
    (6, 32, 128, 64, 1, 32, 32),
    # rows shorter than 64 pixels: tap-major order, resident halos
    (1, 9, 7, 32, 0, 0, 32),       # an image smaller than a tile
    (2, 17, 63, 16, 0, 32, 48),    # two sources, 16-channel slabs
    (1, 34, 26, 160, 1, 128, 144),  # upsampled + skip, one halo buffer; 288 inputs: several output tiles
    (1, 20, 30, 48, 1, 0, 32),     # upsampled source alone, 16-channel slabs
    (24, 32, 32, 96, 0, 0, 128),   # several tiles per CTA: halos, rings and accumulators wrap
]


def bits(x):
    f = U.to_bf16(x).astype(np.float32)
    return (f.view(np.uint32) >> 16).astype(np.uint16)


def val(b):
    return (b.astype(np.uint32) << 16).view(np.float32).astype(np.float64)


def inputs(c, seed):
    N, H, W, C1, up, C2, Cout = c
    rng = np.random.RandomState(seed)
    x1 = bits(np.maximum(rng.normal(size=(N, H // 2, W // 2, C1) if up else (N, H, W, C1)), 0.0))
    x2 = bits(np.maximum(rng.normal(size=(N, H, W, C2)), 0.0)) if C2 else None
    w = bits(rng.normal(0, np.sqrt(2.0 / (9 * (C1 + C2))), (Cout, 9, C1 + C2)))
    x = U.upsample2(val(x1)) if up else val(x1)
    if C2:
        x = np.concatenate([x, val(x2)], 3)
    dout = bits(rng.normal(size=(N, H, W, Cout)))
    return x1, x2, w, x, dout, rng.normal(0, 0.1, Cout).astype(np.float32)


@pytest.mark.parametrize("c", CASES)
def test_forward(ctx, c):
    x1, x2, w, x, _, b = inputs(c, 1)
    out = ctx.conv3x3_fwd(x1, w, c[6], x2=x2, up1=bool(c[4]), bias=b, relu=True)
    ref = np.maximum(U.conv3x3(x, val(w).reshape(c[6], 3, 3, -1), b.astype(np.float64)), 0.0)
    np.testing.assert_allclose(out, ref, rtol=1e-4, atol=1e-5 * np.abs(ref).max())


@pytest.mark.parametrize("c", CASES)
def test_data_gradient(ctx, c):
    x1, x2, w, x, dout, _ = inputs(c, 2)
    wt = np.ascontiguousarray(w.transpose(2, 1, 0))
    din = ctx.conv3x3_dgrad(dout, wt, x1, x2=x2, up1=bool(c[4]), mask_relu=True)
    ref = np.where(x > 0.0, U.conv3x3_dgrad(val(dout), val(w).reshape(c[6], 3, 3, -1)), 0.0)
    np.testing.assert_allclose(val(din), ref, rtol=2.0 ** -7, atol=1e-5 * np.abs(ref).max())


WGRAD_CASES = CASES + [
    (1, 16, 8, 24, 0, 8, 16),       # channel counts that leave part of a group (and 16-output blocks)
    (2, 12, 20, 40, 1, 24, 48),     # the same, expanded from half resolution
    (1, 40, 48, 64, 0, 0, 256),     # eight output blocks: 16-channel groups
    (9, 32, 32, 160, 1, 128, 128),  # several runs per CTA on one set of accumulators
    (10, 128, 128, 16, 0, 0, 32),   # several runs alternating between two sets
]


@pytest.mark.parametrize("c", WGRAD_CASES)
def test_weight_gradient(ctx, c):
    x1, x2, _, x, dout, _ = inputs(c, 3)
    dw = ctx.conv3x3_wgrad(dout, x1, x2=x2, up1=bool(c[4]))
    ref, _ = U.conv3x3_wgrad(x, val(dout))
    ref = ref.reshape(c[6], 9, -1)
    np.testing.assert_allclose(dw, ref, rtol=1e-4, atol=1e-5 * np.abs(ref).max())


@pytest.mark.parametrize("shape", [(1, 64, 80), (2, 80, 144)])
def test_network_gradients(ctx, shape):
    """The whole network at sizes whose upper levels take the tile kernels
    (the data gradients of the decoder write their two sources directly): no
    layer's gradient further from exact FP64 than twice what BF16 storage
    itself moves it, as for the narrow network."""
    N, H, W = shape
    rng = np.random.RandomState(H + W)
    raw = np.zeros((N, H, W, 11), np.float32)
    raw[..., :3] = rng.exponential(0.6, (N, H, W, 3))
    raw[..., 3:10] = rng.uniform(0, 1, (N, H, W, 7))
    raw[..., 10] = 16.0
    target = (raw[..., :3] * rng.uniform(0.5, 1.5, (N, H, W, 3))).astype(np.float32)
    ctx.dn_init(5)
    p = U.init_params(9).astype(np.float32)
    ctx.dn_set_params(p)
    loss = ctx.dn_loss_grads(raw, target)
    g = ctx.dn_get_grads()
    lo, go = U.UNet(p.astype(np.float64), bf16=True).loss_and_grads(raw, target)
    _, gf = U.UNet(p.astype(np.float64), bf16=False).loss_and_grads(raw, target)
    assert abs(loss - lo) <= 1e-4 * lo
    rel = lambda a, b: np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30)  # noqa: E731
    for i, r in enumerate(U.layer_table()[0]):
        for off, n in ((r["w_off"], r["cout_pad"] * 9 * r["cin_pad"]), (r["b_off"], r["cout_pad"])):
            a, b, c = g[off:off + n], go[off:off + n], gf[off:off + n]
            assert rel(a, c) <= 2.0 * rel(b, c) + 2e-3, (i, rel(a, c), rel(b, c))


def _passes(seed, H, W):
    rng = np.random.RandomState(seed)
    rad = rng.exponential(0.6, (H, W, 3)).astype(np.float32)
    rad[rng.uniform(size=(H, W)) < 0.02] = np.nan  # the renderer's rare bad pixels
    rad[rng.uniform(size=(H, W)) < 0.02, 0] = np.inf
    alb, nrm = (rng.uniform(0, 1, (H, W, 3)).astype(np.float32) for _ in range(2))
    dep = np.repeat(rng.uniform(0, 1, (H, W, 1)), 3, 2).astype(np.float32)
    return rad, alb, nrm, dep


@pytest.mark.parametrize("shape", [(33, 64), (50, 130), (17, 40)])
def test_denoise_frame_and_padding(ctx, shape):
    """A frame of any size (the filters fused with the output layer from 64
    padded columns on, separate below) equals the FP64 network on the padded
    record with its filters clamped to the frame: 2e-2 of the largest value,
    what BF16 storage moves the network by; and an output that overlaps the
    radiance gives the same bits."""
    import torch
    H, W = shape
    ctx.dn_init(5)
    p = U.init_params(4).astype(np.float32)
    ctx.dn_set_params(p)
    rad, alb, nrm, dep = _passes(H, H, W)
    out = ctx.denoise(rad, alb, nrm, dep, 8)
    Hp, Wp = (H + 15) // 16 * 16, (W + 15) // 16 * 16
    raw = np.zeros((1, Hp, Wp, 11), np.float32)
    raw[0, :H, :W] = np.concatenate([rad, alb, nrm, dep[..., :1], np.full((H, W, 1), 8, np.float32)], -1)
    logits = U.UNet(p.astype(np.float64), bf16=True).forward(raw)[:, :H, :W]
    ref = U.kp_apply(logits, raw[:, :H, :W])[0]
    fin = np.abs(ref) < 1e4  # +inf reads 65504: its neighbourhood is judged relatively
    np.testing.assert_allclose(out[fin], ref[fin], rtol=2e-2, atol=2e-2 * np.abs(ref[fin]).max())
    np.testing.assert_allclose(out[~fin], ref[~fin], rtol=0.1)
    dev = [torch.from_numpy(x).cuda() for x in (rad, alb, nrm, dep)]
    torch.cuda.synchronize()
    ctx.denoise(*dev, 8, out=dev[0])
    assert np.array_equal(dev[0].cpu().numpy(), out)


@pytest.mark.parametrize("shape", [(1, 48, 64), (2, 80, 144), (1, 32, 48)])
def test_inference_matches_oracle(ctx, shape):
    N, H, W = shape
    ctx.dn_init(5)
    p = U.init_params(6).astype(np.float32)
    ctx.dn_set_params(p)
    rng = np.random.RandomState(W)
    raw = rng.uniform(0, 1, (N, H, W, 11)).astype(np.float32)
    raw[..., 10] = 4.0
    out = ctx.dn_infer(raw)
    ref = U.UNet(p.astype(np.float64), bf16=True).denoise(raw)
    np.testing.assert_allclose(out, ref, rtol=2e-2, atol=2e-2 * np.abs(ref).max())
