"""Traversal-stack entries: a hand-written chain of ten nodes that push seven
children each needs 70 of them (and one for the instance) and fits; the twelve
nodes of the device-error tests need more than there are."""
import pytest

from test_gpu_device_errors import LEAF, Blob, _rays_along_x, _torus_scene, _trace_status

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("levels", [1, 9, 10, 11])
def test_a_chain_of_full_nodes_fits(device, levels):
    from rtgallery import host

    gs = host.GpuScene(device, _torus_scene())
    blob = Blob(gs.models[0].blas)
    mid = (blob.lo + blob.hi) * 0.5
    whole, behind = (blob.lo, blob.hi), ((mid[0], blob.lo[1], blob.lo[2]), blob.hi)  # entered later by a ray along +x
    for i in range(levels):
        last = i == levels - 1
        blob.write_node(i, [behind if last else whole] + [behind] * 7, [LEAF if last else i + 1] + [LEAF] * 7)
    blob.upload()
    _, status = _trace_status(device, gs, _rays_along_x(32))
    assert status == 0
