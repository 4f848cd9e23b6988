"""Kernels that split a map's work by its size, against the oracle, bit for
bit: direct light with several lanes per lumel."""
import numpy as np
import pytest

from oracle_bind import Oracle
from relight_b200 import scenes

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
