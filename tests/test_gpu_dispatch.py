"""Launch rules by size: what a size rule picks gives the bytes of the general path."""
import ctypes as C

import numpy as np
import pytest

from rtgallery import abi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1496, 1000), (1505, 1003)])  # ray slots just below and above 1.5 M
def test_unset_configuration_renders_the_same_image(device, size):
    from rtgallery import host

    scene = scenes.scene_gallery(*size)
    fresh = host.Device()  # no configuration set: packets for large camera-ray lists
    image, _, stats = host.render(fresh, scene, radiance=False)
    config = abi.RtTraversalConfig(128, 0, 20, 0)
    fresh.check(fresh.lib.rt_ctx_set_traversal_config(fresh.ctx, C.byref(config)))
    per_lane, _, per_lane_stats = host.render(fresh, scene, radiance=False)
    fresh.close()
    assert stats == per_lane_stats and stats["status"] == 0
    assert np.array_equal(image, per_lane)


@pytest.mark.parametrize("count", [1, 31, 33, 3647, 3649, 7300, 20_000, 116_735, 116_737, 130_001])
def test_short_ray_lists(device, count):
    """Ray counts around one ray per warp, and around all lanes of the grid."""
    from oracle import oracle as O
    from rtgallery import host

    scene = scenes.scene_gallery(8, 8)
    gs = host.GpuScene(device, scene)
    rays = scenes.random_rays(count, 5 + count, 16.0)
    hits = host.trace_ray_buffer(device, gs, rays)
    want, _ = O.OracleScene(scene).trace(rays)
    for f in ("t", "u", "v", "instance_id", "geometry_index", "primitive_index"):
        assert (np.asarray(hits[f]).view(np.uint32) == np.asarray(want[f]).view(np.uint32)).all(), f
