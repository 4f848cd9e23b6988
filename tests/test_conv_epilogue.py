"""The convolution's epilogue in each way that its four groups share the tiles:
one, two and four accumulator sets, columns held in registers and stored one
chunk after another, with and without bias and masks, over one tile and many,
with edges inside a tile.  BF16 outputs of FP32 sums, against FP64: 2^-8 of the
value and 2^-8 of the largest."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,w", [(1, 3, 5), (2, 37, 150), (4, 130, 140)])
@pytest.mark.parametrize("ci,ncols", [(16, 16), (32, 32), (16, 48), (96, 32), (64, 64), (32, 96), (32, 128), (96, 160),
                                      (16, 256)])
def test_epilogue_splits(cuda, ci, ncols, n, h, w):
    import torch
    from relight_b200 import denoise as D
    g = torch.Generator(device="cuda").manual_seed(ci + ncols)
    x = torch.randn(n, h, w, ci, device="cuda", generator=g).bfloat16()
    wt = (torch.randn(ncols, ci, 3, 3, device="cuda", generator=g) * 0.1).bfloat16()
    wp = wt.permute(2, 3, 1, 0).reshape(9, ci // 8, 8, ncols).permute(0, 1, 3, 2).contiguous()
    bias = torch.randn(ncols, device="cuda", generator=g)
    ref = torch.nn.functional.conv2d(x.double().permute(0, 3, 1, 2), wt.double(), padding=1).permute(0, 2, 3, 1)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    act = torch.relu(ref + bias.double())
    out = torch.zeros(n, h, w, ncols, dtype=torch.bfloat16, device="cuda")
    D.conv3x3(x, wp, ncols, bias=bias, relu=True, out0=out, err=err)
    mask = torch.randn(n, h, w, ncols, device="cuda", generator=g).bfloat16()
    masked = torch.zeros_like(out)
    D.conv3x3(x, wp, ncols, out0=masked, out0_c0=0, out0_cn=ncols, mask0=mask, err=err)
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    for got, r in ((out, act), (masked, ref * (mask > 0))):
        d = (got.double() - r).abs()
        assert bool((d <= 2.0 ** -8 * (r.abs() + r.abs().max())).all()), float(d.max())
