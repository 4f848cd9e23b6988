"""The warp sort and run-length coding of rl_ff_hemisphere at its sizes'
edges, host and device outputs, against the oracle: bit for bit."""
import ctypes as C

import numpy as np
import pytest

from oracle_bind import Oracle
from relight_b200 import _abi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rays", [1, 31, 32, 33, 64, 65, 128, 129, 256, 300, 512, 513, 1024])
def test_hemisphere_run_lengths(cuda, rays):
    import torch
    from relight_b200.device import Relight
    w = scenes.radiosity_room(size=20)
    rl = Relight()
    ds = rl.device_scene(w.scene)
    g = w.radiancemap._device.download(fields=("flags", "position", "normal"))
    valid = np.nonzero(g["flags"] & 1)[0][5:]  # some texels belong to no patch
    pos, nrm = g["position"][valid], g["normal"][valid]
    n = len(valid)
    pot = np.full(400, -1, np.int32)
    pot[valid] = np.arange(n, dtype=np.int32)
    tabs = (np.array([0], np.int32), np.array([[20, 20]], np.int32), np.array([0], np.int64), pot)
    want = Oracle(w.scene.flat).bind_scene(w.scene).ff_hemisphere(pos, nrm, rays, 100.0, 17, *tabs)
    dp, dn = torch.from_numpy(np.ascontiguousarray(pos)).cuda(), torch.from_numpy(np.ascontiguousarray(nrm)).cuda()
    P = lambda a: C.c_void_p(a.ctypes.data)  # noqa: E731
    nnz = C.c_int64()
    head = (ds.handle, n, dp.data_ptr(), dn.data_ptr(), rays, 100.0, 17, P(tabs[0]), 1, P(tabs[1]), P(tabs[2]), P(pot),
            pot.size)
    L = _abi.lib()
    _abi.check(L.rl_ff_hemisphere(*head, None, None, None, 0, C.byref(nnz), None))
    k = nnz.value
    assert k == len(want[1])
    row, cols, vals = np.zeros(n + 1, np.int64), np.zeros(k, np.int32), np.zeros(k, np.float32)
    _abi.check(L.rl_ff_hemisphere(*head, P(row), P(cols), P(vals), k, C.byref(nnz), None))
    drow = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    dcols, dvals = torch.zeros(k, dtype=torch.int32, device="cuda"), torch.zeros(k, device="cuda")
    _abi.check(L.rl_ff_hemisphere_device(*head, drow.data_ptr(), dcols.data_ptr(), dvals.data_ptr(), k, C.byref(nnz), None))
    for a, b, c in ((row, drow, want[0]), (cols, dcols, want[1]), (vals, dvals, want[2])):
        assert np.array_equal(a, c) and np.array_equal(b.cpu().numpy(), c)
