"""rl_intersect_rays over the 32-byte nodes (and, for detail too fine for their
grid, over the full ones) against rl_trace_segments, which walks the full
nodes: the same triangle and t, bit for bit, for scenes that are flat,
small beside their coordinates, or much finer than their size; for rays from
far outside, along the axes and with no length; and for every split of the
rays among warps.  Any-hit queries meet something exactly where closest ones
do."""
import dataclasses

import numpy as np
import pytest

from relight_b200 import scenes

pytestmark = pytest.mark.gpu


def _scene(kind, builder):
    from relight_b200.device import DeviceScene
    f = scenes.terrain_scene(verts=40, n_boxes=50, size=64, tiles=2).scene.flat
    pos = f.pos.astype(np.float32).copy()
    if kind == "flat":
        pos.reshape(-1, 3)[:, 1] = 2.0
    elif kind == "offset":
        pos.reshape(-1, 3)[:] += np.float32([3000.0, -700.0, 12000.0])
    elif kind == "outlier":   # one triangle 10^5 scene sizes away: the full nodes
        pos.reshape(-1, 3)[np.asarray(f.tris).reshape(-1, 3)[-1]] *= np.float32(1e5)
    p = pos.reshape(-1, 3)
    g = dataclasses.replace(f, pos=pos, bounds_lo=p.min(0), bounds_hi=p.max(0))
    return DeviceScene(g, None, builder), f, p


@pytest.mark.parametrize("builder", [0, 1])
@pytest.mark.parametrize("kind", ["plain", "flat", "offset", "outlier"])
def test_packed_walk_equals_full_walk(cuda, kind, builder):
    import torch
    from relight_b200 import _abi
    ds, f, p = _scene(kind, builder)
    L = _abi.lib()
    rng = np.random.default_rng(7)
    lo, hi = np.percentile(p, 0.5, axis=0), np.percentile(p, 99.5, axis=0)
    size = (hi - lo).max()
    for n in (1, 33, 5000, 151553, 700000):   # beyond 151,552 a warp takes several rays a lane
        a, b = rng.uniform(lo - 1, hi + 1, (n, 3)), rng.uniform(lo - 1, hi + 1, (n, 3))
        q = n // 8
        a[:q] = lo + (a[:q] - lo) * 60.0 - 30.0 * size          # from far outside
        axis = rng.integers(0, 3, q)
        b[q:2 * q] = a[q:2 * q]
        b[q + np.arange(q), axis] += rng.choice([-1.0, 1.0], q) * size   # along an axis
        b[2 * q:2 * q + 3] = a[2 * q:2 * q + 3]                 # no length
        seg = np.concatenate([a, b], 1).astype(np.float32)
        d = (seg[:, 3:] - seg[:, :3]).astype(np.float32)
        length = np.sqrt(d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2]).astype(np.float32)
        with np.errstate(all="ignore"):
            d = (d / length[:, None]).astype(np.float32)
        rays = np.zeros((n, 8), np.float32)
        rays[:, :3], rays[:, 3], rays[:, 4:7], rays[:, 7] = seg[:, :3], 0.01, d, length
        T = lambda x: torch.from_numpy(x).cuda()  # noqa: E731
        ds_seg, ds_rays = T(seg), T(rays)
        hit = torch.zeros(n, dtype=torch.int32, device="cuda")
        mf, gp = (torch.zeros((n, 2), dtype=torch.int32, device="cuda") for _ in range(2))
        tuv, tuv2 = (torch.zeros((n, 3), device="cuda") for _ in range(2))
        _abi.check(L.rl_trace_segments(ds.handle, n, ds_seg.data_ptr(), 0, hit.data_ptr(), tuv.data_ptr(), mf.data_ptr(),
                                       None, None, None, None, None))
        _abi.check(L.rl_intersect_rays(ds.handle, n, ds_rays.data_ptr(), 0, gp.data_ptr(), tuv2.data_ptr(), None))
        torch.cuda.synchronize()
        ok = torch.from_numpy(np.isfinite(d).all(1)).cuda()
        assert torch.equal(mf[ok], gp[ok])
        assert torch.equal(tuv[ok][:, 0].view(torch.int32), tuv2[ok][:, 0].view(torch.int32))
        _abi.check(L.rl_intersect_rays(ds.handle, n, ds_rays.data_ptr(), 1, gp.data_ptr(), None, None))
        torch.cuda.synchronize()
        assert torch.equal(gp[ok][:, 0] >= 0, hit[ok] > 0)
        if n == 700000 and kind != "outlier":
            assert int(hit.sum()) > n // 20
