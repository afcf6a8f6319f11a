"""Whose error a call reports.  An error of an asynchronous call comes out of
rtx_synchronize; a synchronous call reports its own alone, also while a replay
of an earlier capture of this context's work, which reports one, is still on
its way; and a batch frame captured by a synchronous call and replayed by an
asynchronous one (or the reverse) reports through the call that replays it.
The errors are traversal stacks of two entries, which stop in bounds.
"""
import pytest

import rendertoy_gb300 as rt
from rendertoy_gb300 import scenes

pytestmark = pytest.mark.gpu

OVERFLOW = "traversal stack overflow"


def _outs(W, H):
    import torch
    return tuple(torch.empty((H, W, 3), device="cuda") for _ in range(3))


def _limit(ctx, n):
    ctx.set_option(rt.OPT_STACK_LIMIT, n)


def test_asynchronous_errors_wait_for_synchronize():
    with rt.Context(0) as ctx:
        ctx.upload(scenes.displaced_icosphere(subdiv=4))
        out = _outs(48, 32)
        ctx.set_option(rt.OPT_ASYNC, 1)
        for bad in (False, True, False):
            _limit(ctx, 2 if bad else 64)
            ctx.aov(48, 32, 700.0, 1500.0, out=out)
            if bad:
                with pytest.raises(rt.RtxError, match="asynchronous"):
                    ctx.synchronize()
            else:
                ctx.synchronize()
        # a host result makes the call synchronous: its error is its own
        _limit(ctx, 2)
        with pytest.raises(rt.RtxError, match=OVERFLOW):
            ctx.aov(48, 32, 700.0, 1500.0)
        # a later call that succeeds clears what an asynchronous one left
        ctx.aov(48, 32, 700.0, 1500.0, out=out)
        _limit(ctx, 64)
        ctx.set_option(rt.OPT_ASYNC, 0)
        ctx.aov(48, 32, 700.0, 1500.0, out=out)
        ctx.synchronize()


def test_replayed_capture_keeps_its_error_to_itself():
    import torch
    s = torch.cuda.Stream()
    with rt.Context(0) as ctx:
        ctx.upload(scenes.displaced_icosphere(subdiv=4))
        ctx._check(ctx.L.rtx_set_stream(ctx.h, s.cuda_stream))
        out, mine = _outs(48, 32), _outs(48, 32)
        ctx.aov(48, 32, 700.0, 1500.0, out=out)
        ctx.set_option(rt.OPT_ASYNC, 1)
        _limit(ctx, 2)
        g = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(g, stream=s, capture_error_mode="relaxed"):
            ctx.aov(48, 32, 700.0, 1500.0, out=out)
        ctx.set_option(rt.OPT_ASYNC, 0)
        _limit(ctx, 64)
        ctx.aov(48, 32, 700.0, 1500.0, out=mine)
        for _ in range(2):
            with torch.cuda.stream(s):
                torch.cuda._sleep(20_000_000)  # some 10 ms before the replay runs
                g.replay()
            ctx.aov(48, 32, 700.0, 1500.0, out=mine)  # must not report the replay's error
        _limit(ctx, 2)
        with pytest.raises(rt.RtxError, match=OVERFLOW):
            ctx.aov(48, 32, 700.0, 1500.0, out=mine)
        torch.cuda.synchronize()
        del g


@pytest.mark.parametrize("first", [0, 1])
def test_batch_graph_reports_through_its_caller(first):
    import torch
    jobs = [dict(scene=0, W=32, H=24, spp=1, seed=1)]
    with rt.Context(0) as ctx:
        ctx.batch_upload([scenes.displaced_icosphere(subdiv=4)])
        out = torch.empty(32 * 24 * 3, device="cuda")
        ctx.set_option(rt.OPT_GRAPH, 1)
        _limit(ctx, 2)
        for mode in (first, 1 - first, first, 1 - first):
            ctx.set_option(rt.OPT_ASYNC, mode)
            for _ in range(2):  # launches and captures, then replays
                if mode:
                    ctx.render_batch(jobs, 4, out=out)
                    with pytest.raises(rt.RtxError, match="asynchronous"):
                        ctx.synchronize()
                else:
                    with pytest.raises(rt.RtxError, match=OVERFLOW):
                        ctx.render_batch(jobs, 4, out=out)
