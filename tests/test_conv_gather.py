"""Forward and data-gradient convolutions of channel counts the tile kernels do
not take -- sources that are a multiple of 8 but not of 16, outputs of a
gradient likewise, more than 512 inputs at narrow rows -- against the FP64
oracle on the same BF16 values: the row kernel (rows of 64 pixels or more, the
inputs together a multiple of 16; resident weights and each depth of the
streamed ring) and the gather kernels (each depth).  Tolerances as for the tile
kernels.
"""
import numpy as np
import pytest

from oracle import unet_oracle as U
from test_conv_tiles import inputs, val

pytestmark = pytest.mark.gpu

FORWARD = [  # N, H, W, C1, up1, C2, Cout
    (1, 5, 64, 24, 0, 8, 32),      # row kernel, resident weights
    (2, 4, 131, 8, 0, 24, 16),     # a second row tile of three pixels
    (1, 6, 128, 24, 1, 40, 64),    # upsampled + skip
    (1, 3, 200, 72, 0, 56, 64),    # streamed weights, six stages
    (1, 3, 70, 40, 0, 24, 128),    # four
    (1, 2, 64, 24, 0, 8, 256),     # two
    (80, 4, 256, 24, 0, 8, 32),    # several tiles per CTA
    (1, 9, 64, 24, 0, 0, 32),      # gather: inputs no multiple of 16
    (1, 20, 20, 24, 0, 8, 32),     # gather: narrow rows, three stages
    (2, 18, 26, 40, 1, 8, 160),    # few CTAs of a wide output: four stages
    (20, 32, 32, 24, 0, 0, 160),   # many: two
    (1, 6, 10, 528, 0, 0, 16),     # more inputs than a resident halo holds
    (1, 1, 1, 8, 0, 0, 16),
]


@pytest.mark.parametrize("c", FORWARD)
def test_forward(ctx, c):
    x1, x2, w, x, _, b = inputs(c, 31)
    out = ctx.conv3x3_fwd(x1, w, c[6], x2=x2, up1=bool(c[4]), bias=b, relu=True)
    ref = np.maximum(U.conv3x3(x, val(w).reshape(c[6], 3, 3, -1), b.astype(np.float64)), 0.0)
    np.testing.assert_allclose(out, ref, rtol=1e-4, atol=1e-5 * np.abs(ref).max())


GRADIENT = [
    (1, 7, 64, 32, 0, 0, 8),       # outputs no multiple of 16: gather, three stages
    (2, 9, 33, 24, 0, 8, 24),      # two sources, narrow rows
    (1, 18, 26, 96, 1, 64, 40),    # upsampled + skip: four stages (few CTAs)
    (20, 32, 32, 160, 0, 0, 24),   # many CTAs: two
    (1, 8, 70, 272, 0, 0, 8),      # two channel tiles
    (1, 6, 10, 32, 0, 0, 528),     # more outputs than a resident halo holds
    (1, 1, 1, 16, 0, 0, 8),
    (1, 12, 72, 24, 0, 8, 32),     # a tile kernel: sources that split inside 16 channels
]


@pytest.mark.parametrize("c", GRADIENT)
@pytest.mark.parametrize("mask", [True, False])
def test_data_gradient(ctx, c, mask):
    x1, x2, w, x, dout, _ = inputs(c, 32)
    wt = np.ascontiguousarray(w.transpose(2, 1, 0))
    din = ctx.conv3x3_dgrad(dout, wt, x1, x2=x2, up1=bool(c[4]), mask_relu=mask)
    ref = U.conv3x3_dgrad(val(dout), val(w).reshape(c[6], 3, 3, -1))
    if mask:
        ref = np.where(x > 0.0, ref, 0.0)
    np.testing.assert_allclose(val(din), ref, rtol=2.0 ** -7, atol=1e-5 * np.abs(ref).max())
