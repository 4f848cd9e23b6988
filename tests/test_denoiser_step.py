"""The denoiser's optimiser step and its in-place inputs and outputs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(n, p, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.rand(n, p, p, 16, generator=g, device="cuda")
    x[..., 10:] = 0
    t = torch.rand(n, p, p, 4, generator=g, device="cuda")
    t[..., :3] += 2.0
    t[..., 3] = (t[..., 3] < 0.8).float()
    return x.to(torch.bfloat16).contiguous(), t.contiguous()


@pytest.mark.parametrize("n,p", [(1, 8), (2, 24), (3, 33)])
def test_adam_and_packed_operands(cuda, n, p):
    """Two Adam steps against numpy on the kernels' own gradients (the float
    atomics of two gradient passes may differ in their last bits: 1e-3 of the
    step), and the operands packed by the step against a fresh packing of the
    same parameters, bit for bit."""
    from relight_b200.denoise import Denoiser
    dn, ref = Denoiser(seed=5), Denoiser(seed=5)
    x, t = _batch(n, p, 3)
    m = v = 0.0
    lr = 1e-3
    for step in (1, 2):
        ref.set_params(dn.params())
        ref.train_step(x, t, lr=-1.0)
        g = ref.grads().astype(np.float64)
        want = dn.params().astype(np.float64)
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        want -= lr * (m / (1 - 0.9 ** step)) / (np.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
        dn.train_step(x, t, lr=lr)
        got = dn.params()
        moved = np.abs(g) > 1e-4 * np.abs(g).max()  # below, rounding decides the sign of g
        assert np.abs(got - want)[moved].max() <= 1e-3 * lr + 1e-7
        assert np.abs(got - want).max() <= 2.5 * lr
    fresh = Denoiser(seed=1)
    fresh.set_params(dn.params())
    assert np.array_equal(dn.forward(x).float().cpu().numpy(), fresh.forward(x).float().cpu().numpy())
    assert dn.status() == 0 and ref.status() == 0


def test_forward_takes_any_placement(cuda):
    """Features and output that are 16-byte aligned (read and written where
    they are), that are not (copied), and the same buffer for both."""
    import ctypes as C
    import torch
    from relight_b200 import _abi
    from relight_b200.denoise import Denoiser
    dn = Denoiser(seed=7)
    x, _ = _batch(1, 40, 9)
    want = dn.forward(x).clone()
    k = x.numel()
    room = torch.zeros(k + 64, dtype=torch.bfloat16, device="cuda")
    for xo, yo in ((1, 0), (0, 3), (5, 2)):
        xs = room[xo:xo + k]
        xs.copy_(x.reshape(-1))
        out = torch.empty(k + 64, dtype=torch.bfloat16, device="cuda")
        y = out[yo:yo + k]
        _abi.check(_abi.lib().rl_denoiser_forward(dn.handle, C.c_void_p(xs.data_ptr()), 1, 40, 40,
                                                  C.c_void_p(y.data_ptr()), None))
        assert torch.equal(y.view_as(want)[..., :3], want[..., :3])
    same = x.clone()
    _abi.check(_abi.lib().rl_denoiser_forward(dn.handle, C.c_void_p(same.data_ptr()), 1, 40, 40,
                                              C.c_void_p(same.data_ptr()), None))
    assert torch.equal(same[..., :3], want[..., :3])


@pytest.mark.parametrize("n,h,w", [(1, 16, 16), (3, 160, 72)])
def test_masked_gradient_columns(cuda, n, h, w):
    """A data gradient of 32 channels into 128 columns of which 96 are kept, in
    one tile per CTA and in several, against
    FP64; BF16 outputs of sums of 288 products: 2^-8 of the value and 2^-8 of
    the largest."""
    import torch
    from relight_b200 import denoise as D
    g = torch.Generator(device="cuda").manual_seed(h)
    x = torch.randn(n, h, w, 32, device="cuda", generator=g).bfloat16()
    wt = (torch.randn(128, 32, 3, 3, device="cuda", generator=g) * 0.1).bfloat16()
    wp = wt.permute(2, 3, 1, 0).reshape(9, 4, 8, 128).permute(0, 1, 3, 2).contiguous()
    m0, m1 = (torch.randn(n, h, w, c, device="cuda", generator=g).bfloat16() for c in (64, 32))
    o0, o1 = torch.zeros_like(m0), torch.zeros_like(m1)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    D.conv3x3(x, wp, 128, out0=o0, out0_c0=0, out0_cn=64, mask0=m0, out1=o1, out1_c0=64, out1_cn=32, mask1=m1, err=err)
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    ref = torch.nn.functional.conv2d(x.double().permute(0, 3, 1, 2), wt.double(), padding=1).permute(0, 2, 3, 1)
    for got, r in ((o0, ref[..., :64] * (m0 > 0)), (o1, ref[..., 64:96] * (m1 > 0))):
        d = (got.double() - r).abs()
        assert bool((d <= 2.0 ** -8 * (r.abs() + r.abs().max())).all()), float(d.max())
