"""Ambient occlusion and final gather through the patch kernels (one warp per
patch of lumels, a shared list of subtrees) against the plain walk from the
root (the opt-in lumel pool), bit for bit: the single calls (patches of one
lumel on these small maps) and the batch (patches of eight), over sample
counts around the chunk of 256 rays and the warp, ray lengths from nothing to
far past the scene, backward rays, sparse iterators and both tree builders."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bake(ds, lm, pms, samples, dist, iterator, how):
    from relight_b200 import _abi, autotune, batch
    from relight_b200.api import AmbientOcclusionSettings, IndirectLightSettings
    lm.upload(color=np.full((lm.width * lm.height, 3), 0.5, np.float32))
    ao = AmbientOcclusionSettings(samples, 0.8, dist, 1.0)
    fg = IndirectLightSettings(1, 1, 0.05, 10.0, samples, dist, 3, (0.5, 0.6, 0.8), (0.01, 0.02, 0.03))
    jobs = [batch.BakeJob.ambient_occlusion(ds, lm, ao, seed=3, iterator=iterator),
            batch.BakeJob.indirect(ds, lm, pms, fg, seed=4, iterator=iterator)]
    if how == "batch":
        b = batch.Batch(jobs)
        b.launch()
        b.close()
    else:
        # the pooled AO walk is the one without a lane split
        saved, split = autotune.get_pool(), C.c_int()
        _abi.check(_abi.lib().rl_tune_get(_abi.TUNE_AO_SPLIT, C.byref(split)))
        if how == "walk":
            autotune.set_pool(1, 32)
            _abi.check(_abi.lib().rl_tune_set(_abi.TUNE_AO_SPLIT, 1))
        try:
            batch.run_per_job(jobs)
        finally:
            autotune.set_pool(*saved)
            _abi.check(_abi.lib().rl_tune_set(_abi.TUNE_AO_SPLIT, split.value))
    return lm.download(fields=("color",))["color"]


@pytest.mark.parametrize("builder", [0, 1])
@pytest.mark.parametrize("which", ["terrain", "room"])
def test_patch_rays_match_the_plain_walk(cuda, which, builder):
    from relight_b200 import scenes
    from relight_b200.device import DeviceMap, Relight
    if which == "terrain":
        wl = scenes.terrain_scene(verts=40, n_boxes=30, size=64, tiles=2, passes=1)
        meshes, scene = len(wl.meshes), wl.scene
    else:
        wl = scenes.room_scene(size=48, n_boxes=5)
        meshes, scene = 1, wl.scene
    rl = Relight(builder=builder)
    ds = rl.device_scene(scene)
    pms = [m._device for m in scene.flat.photonmaps]
    if which == "terrain":
        rl.emit_photons(scene, wl.settings, seed=9)
    lm = DeviceMap(0, 37, 29)
    for m in range(meshes):
        lm.add_mesh(ds, m)
    whole, sparse = (0, 0, 1, -1), (0, 3, 7, -1)
    face = (1, 1, 2, 0)
    cases = [(n, d, whole) for n in (1, 5, 32, 100, 255, 256, 257, 520) for d in (2.0, 50.0)]
    cases += [(17, d, whole) for d in (0.0, -3.0, 0.02, 1e4, 1e30)]
    cases += [(40, 50.0, sparse), (40, 50.0, face)]
    for samples, dist, it in cases:
        want = _bake(ds, lm, pms, samples, dist, it, "walk")
        for how in ("single", "batch"):
            got = _bake(ds, lm, pms, samples, dist, it, how)
            assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), (samples, dist, it, how)
    assert ds.status() == 0
    lm.close()


def test_patch_rays_on_odd_geometry(cuda):
    """One triangle, lumels without a normal, and a floor of
    one plane (every ray starts on the plane of all its triangles)."""
    from relight_b200.api import Lightmap, Mesh, Scene
    from relight_b200.device import DeviceMap, Relight
    for n, drop_normals in ((1, False), (12, False), (12, True)):
        src = Mesh.create()
        xs, zs = np.meshgrid(np.arange(n + 1), np.arange(n + 1), indexing="ij")
        pos = np.stack([xs, np.full_like(xs, 3), zs], -1).reshape(-1, 3).astype(np.float32)
        uv = (np.stack([xs, zs], -1).reshape(-1, 2) / n).astype(np.float32)
        i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
        a = (i * (n + 1) + j).reshape(-1)
        idx = np.stack([a, a + n + 1, a + n + 2, a, a + n + 2, a + 1], -1).reshape(-1)
        if n == 1:
            idx = idx[:3]
        nrm = np.tile([0, 0 if drop_normals else 1, 0], (len(pos), 1)).astype(np.float32)
        src.add_faces(pos, nrm, None, uv, idx)
        scene = Scene()
        scene.begin()
        mesh = scene.add_mesh(src)
        lmap = Lightmap(24, 24)
        lmap.add_mesh(mesh)
        scene.end()
        rl = Relight()
        ds = rl.device_scene(scene)
        lm = lmap._device
        for samples, dist in ((16, 5.0), (300, 0.5)):
            want = _bake(ds, lm, [], samples, dist, (0, 0, 1, -1), "walk")
            for how in ("single", "batch"):
                got = _bake(ds, lm, [], samples, dist, (0, 0, 1, -1), how)
                assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), (n, drop_normals, samples, how)
