"""The separable filters, bit for bit against the oracle where their passes can go
wrong: widths that are a multiple of four pixels but not of eight, around the
1,024-pixel row tiles; heights around the 32-row strips; images smaller than
the filter (RenderToy's reflection wraps into the neighbouring row there);
sizes of each remainder, whose first and last window chunks are known at
compile time; NaN and infinite pixels; an image that starts off a 16-byte
boundary or has rows of another length, which take the 4-byte passes.
"""
import numpy as np
import pytest

from helpers import bits

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 17, 18, 19, 20, 21, 22, 24, 27, 29, 32, 49, 101]


def same(gpu, orc, what):
    nan = np.isnan(orc)  # NaN payloads are not portable, their places are
    assert np.array_equal(np.isnan(gpu), nan), what
    assert np.array_equal(bits(gpu)[~nan], bits(orc)[~nan]), what


@pytest.mark.parametrize("shape", [(1, 1), (3, 13), (33, 31), (65, 33), (5, 1023), (9, 1030), (31, 2061), (1, 4), (3, 12), (31, 8), (33, 44), (65, 36), (5, 1020), (2, 1024), (9, 1028),
                                   (32, 2052)])
def test_quad_passes_bit_exact(ctx, oracle, shape):
    import torch
    H, W = shape
    rng = np.random.RandomState(H * 8191 + W)
    img = rng.exponential(0.7, (H, W, 3)).astype(np.float32)
    flat = img.reshape(-1, 3)
    flat[rng.randint(H * W), 0] = np.nan
    flat[rng.randint(H * W), 2] = np.inf
    buf = torch.zeros(H * W * 3 + 1, dtype=torch.float32, device="cuda")
    off = buf[1:].view(H, W, 3)
    off.copy_(torch.from_numpy(img))
    for size in SIZES:
        blur, bloom = oracle.gaussian_blur(img, size, 0.2 * size), oracle.bloom(img, size, 0.2 * size, 0.8)
        same(ctx.gaussian_blur(img, size, 0.2 * size), blur, (shape, size, "blur"))
        same(ctx.bloom(img, size, 0.2 * size, 0.8), bloom, (shape, size, "bloom"))
        if size in (8, 17):
            for src in (off, torch.from_numpy(img).cuda()):
                out = torch.empty_like(src)
                ctx.bloom(src, size, 0.2 * size, 0.8, out=out)
                ctx.synchronize()
                same(out.cpu().numpy(), bloom, (shape, size, "device bloom"))
