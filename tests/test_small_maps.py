"""Kernels that split a map's work by its size, against the oracle, bit for
bit: direct light with several lanes per lumel and the staged photon gather."""
import numpy as np
import pytest

from oracle_bind import LumelMap, Oracle
from relight_b200 import _abi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("textured", [False, True])
@pytest.mark.parametrize("size", [24, 48, 131])
def test_direct_light_lane_groups(cuda, size, textured):
    """Lights of one and of many samples, one that casts no shadow; the whole
    map, a sparse iterator and a face iterator."""
    from relight_b200.device import FaceBakeIterator, LumelBakeIterator, Relight, lumels
    rl = Relight()
    w = scenes.room_scene(size=size, textured=textured)
    w.scene.flat.lights[1]["casts_shadow"] = 0
    orc = Oracle(w.scene.flat).bind_scene(w.scene)
    ds = rl.device_scene(w.scene)
    for it, spec in ((None, (0, 1, None)), (LumelBakeIterator(2, 3), (2, 3, None)), (FaceBakeIterator(1, 2), (1, 2, 0))):
        w.lightmap._device.clear(colors=True)
        rl.bake_direct_light(w.scene, w.mesh, iterator=it)
        got = lumels(w.lightmap)["color"]
        lm = orc.maps()[0]
        orc.bake_direct(lm, *spec)
        assert lm.color.any() or size == 24
        assert np.array_equal(got.view(np.uint32), lm.color.view(np.uint32)), spec
    assert ds.status() == 0


@pytest.mark.parametrize("W,H,radius", [(64, 64, 7), (65, 63, 7), (130, 70, 0), (70, 66, 3), (40, 33, 15), (40, 33, 16)])
def test_photon_gather_tiles(cuda, W, H, radius):
    """Edges of the 64 x 8 tiles and of the radii that are staged, with
    negative colours and texels without photons."""
    from relight_b200.device import DeviceMap
    rng = np.random.default_rng(W * 100 + H + radius)
    n = W * H
    pm = LumelMap(W, H)
    pm.color[:] = rng.uniform(-1, 2, (n, 3))
    pm.photons[:] = rng.integers(0, 3, n) * (rng.random(n) < 0.3)
    m = DeviceMap(1, W, H)
    m.upload(color=pm.color, photons=pm.photons)
    _abi.check(_abi.lib().rl_photonmap_gather(m.handle, radius, None))
    got = m.download(fields=("gathered",))["gathered"]
    Oracle(scenes.room_scene(size=16).scene.flat).gather(pm, radius)
    assert np.array_equal(got.view(np.uint32), pm.gathered.view(np.uint32))
    m.close()
