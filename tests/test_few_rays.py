"""Small batches of rays and segments, which walk the 4-wide nodes, against
large batches of the same, which do not: the
same triangle, t, u and v, bit for bit, on both builders (the device-built tree
has no 4-wide nodes), for sizes around a warp and around the largest that takes
this path, and in a scene of one triangle."""
import dataclasses

import numpy as np
import pytest

from relight_b200 import scenes

pytestmark = pytest.mark.gpu
FEW = 148 * 32 * 32


def _rays(f, n, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    lo, hi = (torch.tensor(np.asarray(v, np.float32), device="cuda") for v in (f.bounds_lo, f.bounds_hi))
    d = torch.nn.functional.normalize(torch.randn(n, 3, generator=g, device="cuda"), dim=1)
    d[::7, 0] = 0.0
    return torch.cat([lo + (hi - lo) * torch.rand(n, 3, generator=g, device="cuda"),
                      torch.full((n, 1), 0.01, device="cuda"), d, torch.full((n, 1), 300.0, device="cuda")], 1).contiguous()


@pytest.mark.parametrize("builder", [0, 1])
@pytest.mark.parametrize("which", ["terrain", "triangle"])
def test_few_equal_many(cuda, which, builder):
    import torch
    from relight_b200 import _abi
    from relight_b200.device import DeviceScene
    f = scenes.terrain_scene(verts=40, n_boxes=60, size=64, tiles=2).scene.flat
    if which == "triangle":
        first = np.minimum(f.mesh_first_tri, 1).astype(f.mesh_first_tri.dtype)
        f = dataclasses.replace(f, tris=f.tris[:1].copy(), mesh_first_tri=first)
    ds = DeviceScene(f, None, builder)
    L = _abi.lib()
    rays = _rays(f, FEW + 1, 3)
    many, tuv = torch.zeros(FEW + 1, 2, dtype=torch.int32, device="cuda"), torch.zeros(FEW + 1, 3, device="cuda")
    _abi.check(L.rl_intersect_rays(ds.handle, FEW + 1, rays.data_ptr(), 0, many.data_ptr(), tuv.data_ptr(), None))
    for n in (1, 31, 33, 5000, FEW):
        gp, tu = torch.zeros(n, 2, dtype=torch.int32, device="cuda"), torch.zeros(n, 3, device="cuda")
        _abi.check(L.rl_intersect_rays(ds.handle, n, rays.data_ptr(), 0, gp.data_ptr(), tu.data_ptr(), None))
        torch.cuda.synchronize()
        assert torch.equal(gp, many[:n]) and torch.equal(tu.view(torch.int32), tuv[:n].view(torch.int32))
        _abi.check(L.rl_intersect_rays(ds.handle, n, rays.data_ptr(), 1, gp.data_ptr(), None, None))
        torch.cuda.synchronize()
        assert torch.equal(gp[:, 0] >= 0, many[:n, 0] >= 0)
        seg = torch.cat([rays[:n, :3], rays[:n, :3] + 300.0 * rays[:n, 4:7]], 1).contiguous()
        big = seg.repeat(FEW // n + 2, 1)[:FEW + 1].contiguous()   # the same segments over the binary nodes
        out = []
        for s in (seg, big):
            k = len(s)
            hit, mf = torch.zeros(k, dtype=torch.int32, device="cuda"), torch.zeros(k, 2, dtype=torch.int32, device="cuda")
            t3, pt = torch.zeros(k, 3, device="cuda"), torch.zeros(k, 3, device="cuda")
            _abi.check(L.rl_trace_segments(ds.handle, k, s.data_ptr(), 15, hit.data_ptr(), t3.data_ptr(), mf.data_ptr(),
                                           pt.data_ptr(), None, None, None, None))
            torch.cuda.synchronize()
            out.append([x[:n].contiguous().view(torch.int32) for x in (hit, mf, t3, pt)])
        assert all(torch.equal(a, b) for a, b in zip(*out))
    if which == "terrain":
        assert int((many[:, 0] >= 0).sum()) > 1000
