"""The ray sort's two block sizes around the wave (2^20 paths) that separates
them, with queues of whole and ragged chunks: images equal the unsorted ones
bit for bit.
"""
import numpy as np
import pytest

from helpers import bits
from rendertoy_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W, H, spp", [(64, 64, 1), (1024, 1023, 1), (1024, 1024, 1), (1025, 1024, 1), (1024, 1024, 3)])
def test_sorted_equals_unsorted(ctx, W, H, spp):
    import rendertoy_gb300 as rt
    old = ctx.get_option(rt.OPT_SORT_RAYS)
    got = []
    try:
        ctx.upload(scenes.displaced_icosphere(subdiv=3))
        for on in (0, 1):
            ctx.set_option(rt.OPT_SORT_RAYS, on)
            got.append(ctx.render_pt(W, H, spp, 4, seed=6))
    finally:
        ctx.set_option(rt.OPT_SORT_RAYS, old)
    assert np.array_equal(bits(got[0]), bits(got[1]))
