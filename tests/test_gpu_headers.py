"""A built structure's header does not depend on what its buffer held before."""
import ctypes as C

import numpy as np
import pytest

from rtgallery import abi, scenes

pytestmark = pytest.mark.gpu

FIELDS = 132    # bytes of the header up to and with dop_count; the vertices behind it are dop_count many
DOP_COUNT = 32  # its word


@pytest.mark.parametrize("n", [0, 1, 2, 17, 1023, 1024, 1025])
@pytest.mark.parametrize("flags", [abi.RT_BUILD_PREFER_FAST_TRACE, abi.RT_BUILD_PREFER_FAST_BUILD],
                         ids=["trace", "build"])
def test_tlas_header(device, n, flags):
    import torch

    from rtgallery import host

    gs = host.GpuScene(device, scenes.scene_small(8, 8))
    rng = np.random.default_rng(n)
    xf = np.stack([scenes.affine(np.eye(3), rng.uniform(-4, 4, 3), 0.2) for _ in range(max(n, 1))])
    records = gs.patch_instances(scenes.instance_records(xf, np.zeros(len(xf)), np.zeros(len(xf)), 0))
    instances = host.Device.upload(records)
    flags |= abi.RT_BUILD_ALLOW_UPDATE
    sizes = abi.RtBuildSizes()
    device.check(device.lib.rt_get_tlas_build_sizes(n, flags, C.byref(sizes)))
    headers = []
    for fill in (0x00, 0xFF, 0xAB):
        dst = torch.full((sizes.acceleration_structure_size,), fill, dtype=torch.uint8, device="cuda")
        scratch = torch.full((sizes.build_scratch_size,), fill, dtype=torch.uint8, device="cuda")
        device.check(device.lib.rt_cmd_build_tlas(device.ctx, instances.data_ptr(), n, flags, dst.data_ptr(),
                                                  dst.numel(), scratch.data_ptr(), scratch.numel(),
                                                  device.stream_handle()))
        torch.cuda.synchronize()
        headers.append(dst[:FIELDS].cpu().numpy().view(np.uint32))
    assert (headers[0] == headers[1]).all() and (headers[0] == headers[2]).all()
    assert headers[0][DOP_COUNT] == 0


def test_blas_header_keeps_its_vertices(device):
    """A triangle soup's 14-DOP has between 4 and 24 vertices, and they are written."""
    from rtgallery import host

    gs = host.GpuScene(device, scenes.scene_small(8, 8))
    for model in gs.models:
        words = model.blas.buffer[:512].cpu().numpy().view(np.uint32)
        assert 4 <= words[DOP_COUNT] <= 24
