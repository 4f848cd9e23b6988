"""Calls that a program captures replay what the direct call computes: the
blur, whose scratch then is a node of the graph, and a large ray batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(40, 30), (130, 200)])
def test_captured_blur(cuda, w, h):
    import torch
    from relight_b200.device import DeviceMap
    rng = np.random.default_rng(w)
    flags = (rng.random(w * h) < 0.7).astype(np.int32)
    color = rng.random((w * h, 3)).astype(np.float32)
    a, b = DeviceMap(0, w, h), DeviceMap(0, w, h)
    for m in (a, b):
        m.upload(flags=flags, color=color)
    a.blur()
    torch.cuda.synchronize()
    want = a.download(fields=("color",))["color"]
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        b.blur(torch.cuda.current_stream().cuda_stream)
    for _ in range(2):
        b.upload(color=color)
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(b.download(fields=("color",))["color"].view(np.uint32), want.view(np.uint32))


def test_captured_rays(cuda):
    import torch
    from relight_b200 import _abi, scenes
    from relight_b200.device import Relight
    w = scenes.terrain_scene(verts=30, n_boxes=20, size=64, tiles=1)
    ds = Relight().device_scene(w.scene)
    n = 160000
    g = torch.Generator(device="cuda").manual_seed(1)
    lo, hi = (torch.tensor(np.asarray(v, np.float32), device="cuda") for v in (w.scene.flat.bounds_lo, w.scene.flat.bounds_hi))
    d = torch.nn.functional.normalize(torch.randn(n, 3, generator=g, device="cuda"), dim=1)
    rays = torch.cat([lo + (hi - lo) * torch.rand(n, 3, generator=g, device="cuda"), torch.full((n, 1), 0.01, device="cuda"), d,
                      torch.full((n, 1), 300.0, device="cuda")], 1).contiguous()
    want, got = (torch.zeros(n, 2, dtype=torch.int32, device="cuda") for _ in range(2))
    L = _abi.lib()
    _abi.check(L.rl_intersect_rays(ds.handle, n, rays.data_ptr(), 0, want.data_ptr(), None, None))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        _abi.check(L.rl_intersect_rays(ds.handle, n, rays.data_ptr(), 0, got.data_ptr(), None,
                                       torch.cuda.current_stream().cuda_stream))
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want) and bool((want[:, 0] >= 0).any())
