"""The shading kernel's block follows the wave (128, 448 or 896 threads), and no
bit of an image follows the block: frames whose waves sit at the edges of the
rule (2^18 paths; 2^23 with the longer variants) and end in a ragged block,
against the same frame in waves of 2^16 paths, which all take the small block.
"""
import numpy as np
import pytest

from helpers import bits
from rendertoy_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scene, W, H, spp", [("cornell", 512, 511, 1), ("cornell", 512, 512, 1), ("cornell", 513, 512, 1),
                                              ("mixed", 1024, 1023, 8), ("mixed", 1025, 1024, 8)])
def test_block_does_not_change_results(ctx, scene, W, H, spp):
    import rendertoy_gb300 as rt
    ctx.upload(scenes.cornell_box() if scene == "cornell" else scenes.cornell_mixed())
    a = ctx.render_pt(W, H, spp, 4, seed=5)
    ctx.set_option(rt.OPT_WAVE_PATHS, 1 << 16)
    try:
        b = ctx.render_pt(W, H, spp, 4, seed=5)
    finally:
        ctx.set_option(rt.OPT_WAVE_PATHS, 0)
    assert np.array_equal(bits(a), bits(b))


def test_block_does_not_change_batches(ctx):
    import rendertoy_gb300 as rt
    ctx.batch_upload([scenes.cornell_box(), scenes.cornell_mixed()])
    jobs = [dict(scene=0, W=1024, H=1024, spp=4, seed=1), dict(scene=1, W=1025, H=1024, spp=4, seed=2)]
    a = ctx.render_batch(jobs, 4)
    ctx.set_option(rt.OPT_WAVE_PATHS, 1 << 16)
    try:
        b = ctx.render_batch(jobs, 4)
    finally:
        ctx.set_option(rt.OPT_WAVE_PATHS, 0)
    for x, y in zip(a, b):
        assert np.array_equal(bits(x), bits(y))
