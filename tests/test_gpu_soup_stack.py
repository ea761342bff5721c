"""Scattered, heavily overlapping triangles: a ray visits hundreds of nodes, and
a tree a little worse than it need be is too deep for the traversal's stack,
which then reports and loses hits."""
import numpy as np
import pytest

from rtgallery import abi, scenes
from test_gpu_build_edges import TRACE, W4, _scene, _soup

pytestmark = pytest.mark.gpu


def test_three_million_scattered_triangles(device):
    """Every ray's traversal fits the stack, and the hits are those of a tree of another width."""
    from rtgallery import host

    model = _soup(3_000_000, "soup")
    lo, hi = model.positions.min(0), model.positions.max(0)
    rays = scenes.random_rays(262_144, 9, 1.0)
    rays["origin"] = (lo + hi) / 2 + rays["origin"] * (hi - lo)
    rays["tmax"] = 1e30
    hits = []
    for flags in (TRACE, TRACE | W4):
        gs = host.GpuScene(device, _scene(model, scenes.affine(np.eye(3), [0, 0, 0])[None]), blas_flags=flags,
                           tlas_flags=TRACE | abi.RT_BUILD_ALLOW_UPDATE)
        device.read_stats(reset=True)
        hits.append(np.asarray(host.trace_ray_buffer(device, gs, rays, with_models=False)))
        assert device.read_stats(reset=True)["status"] == 0
    assert (hits[0]["instance_id"] == 0).sum() > len(rays) // 2
    assert hits[0].tobytes() == hits[1].tobytes()
