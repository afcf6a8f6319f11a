"""Primary passes and ray queries at the smallest stack the binary walk needs:
the 4-wide walk, which keeps up to three entries a level, must answer them too
(RTX_OPT_STACK_LIMIT lowered; the bound at its full 64 entries is the same
question for deeper trees), with the same hits.
"""
import numpy as np
import pytest

from helpers import bits
from rendertoy_gb300 import scenes

pytestmark = pytest.mark.gpu


def _passes(ctx, rays):
    return [*ctx.primary(40, 30), *ctx.aov(40, 30, 700.0, 1500.0), *ctx.intersect(rays)]


@pytest.mark.parametrize("make", [scenes.cornell_box, scenes.cornell_mixed, lambda: scenes.displaced_icosphere(subdiv=3)])
def test_smallest_binary_stack(ctx, make):
    import rendertoy_gb300 as rt
    rng = np.random.RandomState(3)
    rays = np.concatenate([rng.uniform(-200, 200, (500, 3)), rng.normal(size=(500, 3))], 1).astype(np.float32)
    ctx.upload(make())
    try:
        ctx.set_option(rt.OPT_TRAVERSAL, 0)
        want = _passes(ctx, rays)
        for limit in range(2, 65):
            ctx.set_option(rt.OPT_STACK_LIMIT, limit)
            try:
                _passes(ctx, rays)
                break
            except rt.RtxError as e:
                assert "traversal stack overflow" in str(e)
        assert 2 < limit < 40
        ctx.set_option(rt.OPT_TRAVERSAL, 2)
        for a, b in zip(want, _passes(ctx, rays)):
            assert np.array_equal(a, b) if a.dtype == np.int32 else np.array_equal(bits(a), bits(b))
        ctx.set_option(rt.OPT_STACK_LIMIT, 2)  # neither walk's: still an error
        with pytest.raises(rt.RtxError, match="traversal stack overflow"):
            _passes(ctx, rays)
    finally:
        ctx.set_option(rt.OPT_STACK_LIMIT, 64)
        ctx.set_option(rt.OPT_TRAVERSAL, 2)
