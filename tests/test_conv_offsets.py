"""Convolutions and GEMMs on device tensors that start off a 16-byte boundary
(views into larger tensors): the kernels read and write 16 bytes at a time, so
such operands are staged, and the results equal those of aligned tensors bit
for bit.
"""
import pytest

pytestmark = pytest.mark.gpu


def _view(x, off):
    """A copy of x that starts `off` elements into a fresh buffer."""
    import torch
    buf = torch.zeros(x.numel() + off + 8, dtype=x.dtype, device="cuda")
    v = buf[off:off + x.numel()].view(x.shape)
    v.copy_(x)
    return v


@pytest.mark.parametrize("off", [1, 3, 4])
@pytest.mark.parametrize("c", [
    (1, 20, 64, 32, 0, 0, 32),   # rows of 64 pixels
    (2, 18, 26, 32, 1, 16, 48),  # narrow rows, upsampled + skip
    (1, 9, 66, 24, 0, 8, 16),    # channels that are no multiple of 16 per source
])
def test_operands_off_a_16_byte_boundary(ctx, c, off):
    import torch
    N, H, W, C1, up, C2, Cout = c
    g = torch.Generator(device="cuda").manual_seed(7)

    def r(*s):
        return torch.randn(s, generator=g, device="cuda").to(torch.bfloat16)

    x1 = r(N, H // 2, W // 2, C1) if up else r(N, H, W, C1)
    x2 = r(N, H, W, C2) if C2 else None
    w, wt, dout = r(Cout, 9, C1 + C2), r(C1 + C2, 9, Cout), r(N, H, W, Cout)
    bias = torch.randn(Cout, generator=g, device="cuda")
    res = []
    for k in (0, off):
        ops = [x if k == 0 or x is None else _view(x, k) for x in (
            x1, x2, w, wt, dout, bias, w.view(-1)[:40 * 72].view(40, 72), wt.view(-1)[:48 * 72].view(48, 72),
            torch.zeros((N, H, W, Cout), device="cuda"), torch.zeros((Cout, 9, C1 + C2), device="cuda"),
            torch.zeros((N, H, W, C1 + C2), dtype=torch.bfloat16, device="cuda"), torch.zeros((40, 48), device="cuda"))]
        v1, v2, vw, vwt, vd, vb, ga, gb, out, dw, din, gc = ops
        torch.cuda.synchronize()
        ctx.conv3x3_fwd(v1, vw, Cout, x2=v2, up1=bool(up), bias=vb, relu=True, out=out)
        ctx.conv3x3_dgrad(vd, vwt, v1, x2=v2, up1=bool(up), mask_relu=True, out=din)
        ctx.conv3x3_wgrad(vd, v1, x2=v2, up1=bool(up), out=dw)
        ctx.gemm_bf16(ga, gb, out=gc)
        ctx.synchronize()
        res.append((out.cpu(), din.float().cpu(), dw.cpu(), gc.cpu()))
    for name, a, b in zip(("fwd", "dgrad", "wgrad", "gemm"), *res):
        if name == "wgrad":  # FP32 atomics in any order
            torch.testing.assert_close(a, b, rtol=1e-5, atol=1e-5 * a.abs().max().item())
        else:
            assert torch.equal(a, b), name
