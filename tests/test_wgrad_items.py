"""The weight gradient's split into products of 64 input channels: gradient
channels on both sides of the 64 that one block holds, input channels on both
sides of a block's and beyond one launch's list, rows of dW that start on 16
bytes and that do not, and fewer tiles than there are CTAs to share them.

Tolerance: products of BF16 values summed in FP32 in two orders; 2e-3 of the
largest entry is far above their rounding (2^-24 per term) and far below one
lost or doubled tile."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,w,co,cin,off,total", [
    (1, 8, 16, 64, 64, 0, 64), (1, 9, 17, 65, 65, 0, 128), (3, 5, 3, 3, 16, 4, 24), (2, 40, 50, 32, 130, 0, 192),
    (1, 16, 16, 128, 1100, 1, 1104), (20, 64, 64, 16, 48, 8, 64)])
def test_wgrad_items(cuda, n, h, w, co, cin, off, total):
    import torch
    from relight_b200 import denoise as D
    g = torch.Generator(device="cuda").manual_seed(n + cin)
    gs, cs = (co + 15) // 16 * 16, (cin + 7) // 8 * 8
    grad = torch.zeros(n, h, w, gs, device="cuda", dtype=torch.bfloat16)
    x = torch.randn(n, h, w, cs, device="cuda", generator=g).bfloat16()
    grad[..., :co] = torch.randn(n, h, w, co, device="cuda", generator=g).bfloat16()
    dw = torch.zeros(co, 9, total, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    D.conv3x3_wgrad(grad, co, x, cin, dw, ci_off=off, err=err)
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    ref = torch.nn.grad.conv2d_weight(x.double()[..., :cin].permute(0, 3, 1, 2), (co, cin, 3, 3),
                                      grad.double()[..., :co].permute(0, 3, 1, 2), padding=1)
    ref = ref.permute(0, 2, 3, 1).reshape(co, 9, cin)
    e = (dw[..., off:off + cin] - ref).abs().max().item()
    assert e <= 2e-3 * ref.abs().max().item(), (e, ref.abs().max().item())
    assert not dw[..., :off].any() and not dw[..., off + cin:].any()
