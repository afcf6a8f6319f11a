"""A captured batch frame holds the addresses of the path workspace and of the
job table.  Calls between two equal batches that make either move -- a larger
render, a larger batch launched directly -- must lead to a new capture
(kernel launches instead of a replay), and the frames stay equal to direct
launches bit for bit; calls that move nothing leave the replay in place.
"""
import numpy as np
import pytest

import rendertoy_gb300 as rt
from helpers import bits
from rendertoy_gb300 import scenes

pytestmark = pytest.mark.gpu

JOBS = [dict(scene=0, W=24, H=20, spp=2, seed=1), dict(scene=1, W=17, H=9, spp=3, seed=2)]


def _larger_render(ctx):
    ctx.upload(scenes.cornell_box())
    ctx.render_pt(96, 64, 2, 4, seed=5)


def _larger_batch(ctx):
    # per-kernel timers: launched directly, no graph involved
    ctx.set_option(rt.OPT_KERNEL_TIMING, 1)
    try:
        ctx.render_batch([dict(scene=k % 2, W=40 + k, H=32, spp=2, seed=k) for k in range(12)], 4)
    finally:
        ctx.set_option(rt.OPT_KERNEL_TIMING, 0)


def _more_jobs_same_paths(ctx):
    # 600 frames of one path: the job table alone grows
    ctx.set_option(rt.OPT_KERNEL_TIMING, 1)
    try:
        ctx.render_batch([dict(scene=0, W=1, H=1, spp=1, seed=k) for k in range(600)], 4)
    finally:
        ctx.set_option(rt.OPT_KERNEL_TIMING, 0)


@pytest.mark.parametrize("between, moves", [(_larger_render, True), (_larger_batch, True),
                                            (_more_jobs_same_paths, None), (lambda ctx: None, False)])
def test_moved_buffers_are_captured_anew(between, moves):
    with rt.Context(0) as ctx:  # a fresh workspace: the first batch sizes it
        ctx.batch_upload([scenes.cornell_box(), scenes.cornell_mixed()])
        direct = [f.copy() for f in ctx.render_batch(JOBS, 4)]
        ctx.set_option(rt.OPT_GRAPH, 1)
        ctx.render_batch(JOBS, 4)  # renders and captures
        ctx.render_batch(JOBS, 4)
        assert ctx.stats()["kernel_launches"] == 0
        between(ctx)
        again = ctx.render_batch(JOBS, 4)
        if moves is not None:  # a grown job table may land where the old one was
            assert (ctx.stats()["kernel_launches"] > 0) == moves
        for a, b in zip(direct, again):
            assert np.array_equal(bits(a), bits(b))
        replay = ctx.render_batch(JOBS, 4)
        assert ctx.stats()["kernel_launches"] == 0
        for a, b in zip(direct, replay):
            assert np.array_equal(bits(a), bits(b))
