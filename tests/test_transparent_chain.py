"""Segments through transparent texels, whose first walk is apart from the
ones that go on behind a texel: on the textured room, a large batch and a small
one of the same segments against the oracle tracer, for each set of flags."""
import numpy as np
import pytest

from relight_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [0, 15, 16, 31])
def test_segments_through_cutouts(cuda, flags):
    import torch
    from oracle_bind import Oracle
    from relight_b200 import _abi
    from relight_b200.device import Relight
    w = scenes.room_scene(size=48, textured=True)
    ds = Relight().device_scene(w.scene)
    f = w.scene.flat
    rng = np.random.default_rng(flags)
    seg = np.concatenate([rng.uniform(f.bounds_lo - 1, f.bounds_hi + 1, (20000, 3)),
                          rng.uniform(f.bounds_lo - 1, f.bounds_hi + 1, (20000, 3))], 1).astype(np.float32)
    ref = Oracle(f).bind_scene(w.scene).trace_segments(seg, flags)
    for repeat in (1, 8):   # 160,000: the path of large batches
        s = torch.from_numpy(np.tile(seg, (repeat, 1))).cuda()
        n = len(s)
        hit, mf = torch.zeros(n, dtype=torch.int32, device="cuda"), torch.zeros(n, 2, dtype=torch.int32, device="cuda")
        pt = torch.zeros(n, 3, device="cuda")
        _abi.check(_abi.lib().rl_trace_segments(ds.handle, n, s.data_ptr(), flags, hit.data_ptr(), None, mf.data_ptr(),
                                                pt.data_ptr(), None, None, None, None))
        torch.cuda.synchronize()
        m = ref["hit"] > 0
        for k in range(repeat):
            part = slice(k * 20000, (k + 1) * 20000)
            assert np.array_equal(hit[part].cpu().numpy() > 0, m)
            g = mf[part].cpu().numpy()
            assert np.array_equal(g[m, 0], ref["mesh"][m]) and np.array_equal(g[m, 1], ref["face"][m])
            assert np.array_equal(pt[part].cpu().numpy()[m], ref["point"][m])
