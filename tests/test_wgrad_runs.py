"""Weight gradients over several runs per CTA.  The tensor core truncates when it
adds to an accumulator: about n 2^-26 of the sum after n MMAs of 16 pixels, so
a run is at most as long as its layer's limit R (rows of fewer than 64 pixels:
P / (8 * 152 / ceil(9 Cin / 128)) rounded up to 64 pixels), and the F = P / R
partial sums add up in FP32, 2.6e-8 of the growing sum each (a third of an
ulp), sqrt(F / 3) of them.  With gradients of one sign, so that nothing cancels
and truncation shows, the relative L2 error against FP64 stays below 1.25 times
the sum of the two.  Runs twice to four times as long exceed that.
"""
import numpy as np
import pytest

from oracle import unet_oracle as U
from test_conv_tiles import bits, inputs, val

pytestmark = pytest.mark.gpu


def _limit(N, H, W, Cin):
    P = N * H * W
    ranges = max(1, 8 * 152 // -(-9 * Cin // 128))
    return max(64, -(-(-(-P // ranges)) // 64) * 64)


@pytest.mark.parametrize("c", [
    (8, 32, 32, 96, 1, 64, 64),    # limit 128 pixels
    (32, 32, 32, 64, 0, 0, 64),    # 192
    (8, 62, 62, 64, 0, 0, 64),     # 192, ragged tiles
    (8, 62, 62, 96, 1, 64, 64),    # 320
    (32, 16, 16, 96, 1, 64, 64),   # 128
    (1, 68, 60, 32, 0, 0, 32),     # 64: one tile
])
def test_error_of_sums_of_one_sign(ctx, c):
    N, H, W, C1, up, C2, Cout = c
    x1, x2, _, x, dout, _ = inputs(c, 11)
    dout = bits(np.abs(val(dout)))
    dw = ctx.conv3x3_wgrad(dout, x1, x2=x2, up1=bool(up))
    ref, _ = U.conv3x3_wgrad(x, val(dout))
    ref = ref.reshape(Cout, 9, -1)
    R = _limit(N, H, W, C1 + C2)
    F = -(-N * H * W // R)
    err = np.linalg.norm(dw - ref) / np.linalg.norm(ref)
    bound = 1.25 * (R / 16 * 2.0 ** -26 + 2.6e-8 * np.sqrt(F / 3))
    print(f"{c}: error {err:.3g}, bound {bound:.3g}")
    assert err <= bound


@pytest.mark.parametrize("c", [
    (4, 20, 30, 32, 0, 0, 64),      # two runs of a tile, held in registers
    (32, 16, 16, 128, 0, 0, 160),   # two blocks of outputs held, the last CTA's alone
    (8, 16, 16, 16, 0, 0, 48),      # 16-channel groups, blocks of 16 outputs
    (16, 32, 32, 16, 0, 0, 80),     # the same, several runs
    (6, 100, 68, 64, 1, 32, 32),    # three channel groups shared out over CTAs
    (5, 68, 100, 160, 1, 0, 16),    # five groups, one block of 16 outputs
    (3, 24, 40, 24, 0, 8, 96),      # part-filled groups over several runs
    (16, 40, 24, 96, 0, 0, 256),    # eight blocks of outputs
    (40, 8, 8, 32, 1, 32, 32),      # tiles of one image each, many per CTA
    (200, 2, 6, 32, 0, 0, 32),      # images smaller than a tile
    (2, 272, 96, 64, 0, 0, 64),     # tall tiles, several runs
    (15, 80, 96, 136, 0, 8, 16),    # a ring that fills shared memory
])
def test_splits(ctx, c):
    """Every way a layer is shared out, against the oracle; tolerance as for
    the other tile convolutions."""
    x1, x2, _, x, dout, _ = inputs(c, 12)
    dw = ctx.conv3x3_wgrad(dout, x1, x2=x2, up1=bool(c[4]))
    ref, _ = U.conv3x3_wgrad(x, val(dout))
    ref = ref.reshape(c[6], 9, -1)
    np.testing.assert_allclose(dw, ref, rtol=1e-4, atol=1e-5 * np.abs(ref).max())
