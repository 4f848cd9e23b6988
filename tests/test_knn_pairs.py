"""The k-nearest-neighbour estimate where a warp searches for two neighbouring
lumels at once: bit for bit against the float32 brute force of
oracle/knn_ref.py, on smooth charts with seams, odd widths and holes, in each
split of a row among warps, far from the origin, with pools of records that
overflow a buffer, and with grids of few and of many cells."""
import numpy as np
import pytest

from knn_ref import knn_gather

pytestmark = pytest.mark.gpu


def _chart(w, h, seam, at, rng):
    """A bent sheet; beyond the column `seam` it lies elsewhere."""
    x, z = np.meshgrid(np.arange(w) * 0.11, np.arange(h) * 0.13)
    x = np.where(np.arange(w) >= seam, 9.0 - x, x)
    pos = np.stack([x, np.sin(x) * 0.6 + 0.2 * z, z], -1).reshape(-1, 3).astype(np.float32) + np.float32(at)
    return pos, (rng.random(w * h) < 0.8).astype(np.int32)


@pytest.mark.parametrize("w,h,seam,at,k,radius,cell", [
    (1, 3, 9, 0.0, 5, 1.0, 80), (3, 5, 2, 0.0, 128, 1.5, 80), (9, 40, 4, 0.0, 20, 0.7, 24),
    (17, 33, 8, 4096.0, 100, 1.0, 80), (70, 61, 33, -300.0, 10, 1.5, 80), (70, 61, 33, 0.0, 10, 1.5, 8),
    (700, 90, 351, 0.0, 30, 0.5, 80), (1024, 60, 77, 10.0, 100, 0.6, 128)])
def test_pairs_match_brute_force(cuda, w, h, seam, at, k, radius, cell):
    import torch
    from relight_b200 import autotune
    from relight_b200.device import DeviceMap, PhotonRecords
    rng = np.random.default_rng(w + k)
    pos, flags = _chart(w, h, seam, at, rng)
    if w > 500:   # the brute force on some columns around the seam and the ends
        keep = np.zeros((h, w), bool)
        keep[:, [0, 1, 2, seam - 2, seam - 1, seam, seam + 1, w - 3, w - 2, w - 1]] = True
        keep[h // 2, :] = True
        check_at = keep.reshape(-1) & (flags > 0)
    else:
        check_at = flags > 0
    n = 6000
    near = pos[rng.integers(0, len(pos), n)] + rng.normal(0, 0.2, (n, 3)).astype(np.float32)
    near[:900] = pos[len(pos) // 2] + rng.normal(0, 0.05, (900, 3)).astype(np.float32)   # a pool
    near[900:1300] = near[899]                                                           # ties past every k
    near[1300] = pos[0] + np.float32(300.0)   # a long box: many empty cells
    rec6 = np.concatenate([near, rng.uniform(-1, 1, (n, 3))], 1).astype(np.float32)
    photon, depth = rng.permutation(n).astype(np.uint32), rng.integers(0, 4, n).astype(np.int32)
    slot = (rng.random(n) < 0.1).astype(np.int32)
    pm = DeviceMap(1, w, h)
    pm.upload(flags=flags, position=pos)
    rec = PhotonRecords(n)
    rec.upload(rec6, photon, depth, slot)
    old = autotune.get_knn_cell()
    try:
        autotune.set_knn_cell(cell)
        rec.gather_knn(pm, 0, k, radius)
        torch.cuda.synchronize()
    finally:
        autotune.set_knn_cell(old)
    got = pm.download(fields=("gathered",))["gathered"]
    want = knn_gather(pos, check_at, rec6, photon, depth, slot, 0, k, radius)
    assert np.array_equal(got[check_at].view(np.uint32), want[check_at].view(np.uint32))
    rec.close()
