"""rl_ff_pairwise against the oracle at the edges of its tiles of 32 x 128
patches and of the rows' sort: bit for bit, with coincident patches, normals
that are zero or not unit, and thresholds from none to most."""
import ctypes as C

import numpy as np
import pytest

from oracle_bind import Oracle
from relight_b200 import _abi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 2, 32, 33, 128, 129, 161, 700])
@pytest.mark.parametrize("threshold", [-1.0, 0.0, 0.02, 0.5])
def test_pairwise_edges(cuda, n, threshold):
    import torch
    from relight_b200.device import Relight
    w = scenes.room_scene(size=24, n_boxes=3)
    rl = Relight()
    ds = rl.device_scene(w.scene)
    rng = np.random.default_rng(n)
    pos = rng.uniform(0.2, 3.0, (n, 3)).astype(np.float32)
    nrm = rng.normal(size=(n, 3)).astype(np.float32)
    if n > 40:
        pos[5] = pos[30]            # no distance
        nrm[7] = 0
        nrm[9] *= 100
        nrm[11] *= 1e-3
    want = Oracle(w.scene.flat).bind_scene(w.scene).ff_pairwise(pos, nrm, threshold) if n else None
    dp, dn = torch.from_numpy(pos).cuda(), torch.from_numpy(nrm).cuda()
    count = C.c_int64(-1)
    args = (ds.handle, n, dp.data_ptr(), dn.data_ptr(), threshold)
    L = _abi.lib()
    _abi.check(L.rl_ff_pairwise(*args, None, None, None, 0, C.byref(count), None))
    k = count.value
    assert k == (len(want[1]) if n else 0)
    row, cols, vals = np.zeros(n + 1, np.int64), np.zeros(max(k, 1), np.int32), np.zeros(max(k, 1), np.float32)
    ptr = [C.c_void_p(a.ctypes.data) for a in (row, cols, vals)]
    if k:
        assert L.rl_ff_pairwise(*args, *ptr, k - 1, C.byref(count), None) == 5  # RL_CAPACITY
    _abi.check(L.rl_ff_pairwise(*args, *ptr, k, C.byref(count), None))
    if n:
        assert np.array_equal(row, want[0]) and np.array_equal(cols[:k], want[1])
        # a row of zeros divides by its zero sum: any NaN will do
        same = vals[:k].view(np.uint32) == want[2].view(np.uint32)
        assert (same | (np.isnan(vals[:k]) & np.isnan(want[2]))).all()
