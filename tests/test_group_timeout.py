"""Waits that run out in one warp of a group: the four warps of the fused output
layer's epilogue wait for an accumulator each by itself and share a barrier per
tile, so one whose wait runs out must leave together with the others.  The
diagnostic call makes each warp in turn lose its wait; a warp that left at
another tile than its partners would report "index out of range" beside the
timeout.  The layer itself still gives the oracle's loss afterwards, over
several tiles per group.
"""
import numpy as np
import pytest

from oracle import unet_oracle as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("polls", [1, 64])
def test_group_leaves_together(ctx, polls):
    r = ctx.L.rtx_selftest_wait_timeout(ctx.h, polls)
    assert r == 5, r  # RTX_ERR_DEVICE
    assert ctx.L.rtx_last_error(ctx.h) == b"kernel error: tensor-core barrier wait timed out"
    N, H, W = 5, 128, 256  # 1,280 tiles: more than one per group
    rng = np.random.RandomState(polls)
    raw = rng.uniform(0, 1, (N, H, W, 11)).astype(np.float32)
    raw[..., 10] = 4.0
    ctx.dn_init(5)
    ctx.dn_set_params(U.init_params(4).astype(np.float32))
    one = ctx.dn_infer(raw[:1])
    many = ctx.dn_infer(raw)
    assert np.array_equal(many[:1].view(np.uint32), one.view(np.uint32))
