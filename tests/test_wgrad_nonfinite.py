"""Infinite and NaN activations in weight gradients: only the weights whose
sums read the value become non-finite, as in the FP64 sums (zero padding
outside the image, finite gradients).  Values sit in corners, first and last
rows and columns, and inside, at widths and heights that are and are not a
multiple of a tile, for full-resolution, upsampled and skip sources.
"""
import numpy as np
import pytest

from oracle import unet_oracle as U
from test_conv_tiles import bits, inputs, val

pytestmark = pytest.mark.gpu

CASES = [
    (1, 16, 16, 32, 0, 0, 32),
    (2, 17, 20, 32, 0, 0, 64),     # ragged both ways
    (1, 32, 72, 64, 0, 32, 32),    # three channel groups
    (3, 18, 26, 32, 1, 16, 48),    # upsampled + skip, blocks of 16 outputs
    (4, 24, 40, 16, 0, 0, 32),     # 16-channel groups
    (32, 16, 16, 64, 0, 0, 64),    # several runs per CTA
    (1, 1, 7, 32, 0, 0, 16),       # one row: first and last
]


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("c", CASES)
def test_spreads_no_further(ctx, c, bad):
    N, H, W, C1, up, C2, Cout = c
    x1, x2, _, _, dout, _ = inputs(c, 21)
    v1, v2 = val(x1), None if x2 is None else val(x2)
    h, w = v1.shape[1:3]
    spots = [(0, 0), (0, w // 2), (h - 1, 0), (h - 1, w - 1), (h // 2, w - 1), (h // 2, w // 2), (0, w - 1)]
    for k, (y, x) in enumerate(spots):
        v1[k % N, y, x, 2 * k + 1] = bad
    if v2 is not None:
        v2[N - 1, H - 1, W // 3, 1] = v2[0, 0, W - 1, 4] = bad
    with np.errstate(invalid="ignore"):
        dw = ctx.conv3x3_wgrad(dout, bits(v1), x2=None if v2 is None else bits(v2), up1=bool(up))
        x = U.upsample2(v1) if up else v1
        if v2 is not None:
            x = np.concatenate([x, v2], 3)
        ref, _ = U.conv3x3_wgrad(x, val(dout))
    ref = ref.reshape(Cout, 9, -1)
    assert np.array_equal(np.isnan(dw), np.isnan(ref))
    inf = np.isinf(ref)
    assert np.array_equal(dw[inf], ref[inf])
    fin = np.isfinite(ref)
    assert np.isfinite(dw[fin]).all() and 0 < fin.mean() < 1
    np.testing.assert_allclose(dw[fin], ref[fin], rtol=1e-4, atol=1e-5 * np.abs(ref[fin]).max())


def test_all_nan(ctx):
    """A layer of NaN, as in a diverged training run, ends in time: every
    weight NaN, no wait runs out."""
    N, H, W, C1, Cout = 16, 64, 64, 64, 64
    x1, _, _, _, dout, _ = inputs((N, H, W, C1, 0, 0, Cout), 22)
    dw = ctx.conv3x3_wgrad(dout, np.full_like(x1, 0x7FC0))
    assert np.isnan(dw).all()
    dw = ctx.conv3x3_wgrad(dout, np.full_like(x1, 0x7F80))  # +inf
    assert not np.isfinite(dw).any()
