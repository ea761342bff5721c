"""Launch rules by size: what a size rule picks gives the bytes of the general path."""
import numpy as np
import pytest

from rtgallery import scenes

pytestmark = pytest.mark.gpu


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
