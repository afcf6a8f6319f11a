"""The longest separable filters whose strip of pixels fits shared memory: 568
taps down, 12,493 across.  At and below them a bloom takes two launches (four
on the direct path, from 569 taps on) and the row pass follows
RTX_OPT_COMPOSITOR_FMA; results equal the oracle's bit for bit either way, and
fused ones are within the fused filters' 1e-5 of the sum of magnitudes (here
of the blur itself: all pixels are positive).
"""
import numpy as np
import pytest

from helpers import bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [265, 266, 268, 269, 561, 562, 563, 564, 565, 566, 567, 568, 569])
def test_longest_column_windows(ctx, oracle, size):
    img = np.random.RandomState(size).exponential(0.7, (41, 35, 3)).astype(np.float32)
    got = ctx.bloom(img, size, size / 6.0, 0.8)
    assert ctx.stats()["kernel_launches"] == (2 if size <= 568 else 4)
    assert np.array_equal(bits(got), bits(oracle.bloom(img, size, size / 6.0, 0.8)))


@pytest.mark.parametrize("size", [12489, 12490, 12491, 12492, 12493])
def test_longest_row_windows(ctx, oracle, size):
    import rendertoy_gb300 as rt
    img = np.random.RandomState(size).exponential(0.7, (1, 1033, 3)).astype(np.float32)
    ref = oracle.gaussian_blur(img, size, size / 6.0)
    got = ctx.gaussian_blur(img, size, size / 6.0)
    ctx.set_option(rt.OPT_COMPOSITOR_FMA, 1)
    try:
        fused = ctx.gaussian_blur(img, size, size / 6.0)
    finally:
        ctx.set_option(rt.OPT_COMPOSITOR_FMA, 0)
    assert np.array_equal(bits(got), bits(ref))
    assert not np.array_equal(bits(fused), bits(got))
    np.testing.assert_allclose(fused, ref, rtol=1e-5)


@pytest.mark.parametrize("size", [180, 181, 189, 190, 200, 201, 264, 265, 266, 269, 281])
def test_column_forms_by_strip_size(ctx, oracle, size):
    """Rows of a multiple of four pixels: the 16-byte and the 4-byte column
    passes on both sides of where one gives way to the other."""
    img = np.random.RandomState(size).exponential(0.7, (43, 36, 3)).astype(np.float32)
    assert np.array_equal(bits(ctx.gaussian_blur(img, size, size / 6.0)), bits(oracle.gaussian_blur(img, size, size / 6.0)))
    assert np.array_equal(bits(ctx.bloom(img, size, size / 6.0, 0.8)), bits(oracle.bloom(img, size, size / 6.0, 0.8)))
