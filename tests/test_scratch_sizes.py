"""The sizes that callers query, and keep buffers of, are fixed numbers."""
import ctypes as C

import pytest

from rtgallery import abi

T, B = abi.RT_BUILD_PREFER_FAST_TRACE, abi.RT_BUILD_PREFER_FAST_BUILD
Q, W4 = abi.RT_BUILD_QUANTIZED_NODES, abi.RT_BUILD_EXT_NODE_WIDTH_4

SIZES = [
    # top level, primitives, flags, structure, build scratch, update scratch
    (False, 3, T, 1_536, 24_320, 512),
    (False, 3, B, 1_536, 22_016, 512),
    (False, 3, T | Q, 1_280, 25_088, 512),
    (False, 3, T | W4, 2_048, 24_320, 512),
    (False, 1_025, T, 218_880, 260_608, 37_376),
    (False, 1_025, B, 218_880, 168_448, 37_376),
    (False, 1_025, T | Q, 113_408, 429_568, 37_376),
    (False, 1_025, T | W4, 312_832, 260_608, 37_376),
    (False, 2_000_001, T, 425_144_064, 466_160_640, 72_000_512),
    (False, 2_000_001, B, 425_144_064, 290_150_912, 72_000_512),
    (False, 2_000_001, T | Q, 219_429_632, 795_303_936, 72_000_512),
    (False, 2_000_001, T | W4, 608_001_536, 466_160_640, 72_000_512),
    (True, 3, T, 2_048, 24_832, 512),
    (True, 3, B, 2_048, 22_528, 512),
    (True, 3, T | Q, 2_048, 24_832, 512),
    (True, 3, T | W4, 2_560, 24_832, 512),
    (True, 1_025, T, 303_616, 391_936, 37_376),
    (True, 1_025, B, 303_616, 299_776, 37_376),
    (True, 1_025, T | Q, 303_616, 391_936, 37_376),
    (True, 1_025, T | W4, 399_104, 391_936, 37_376),
    (True, 2_000_001, T, 590_287_104, 722_160_896, 72_000_512),
    (True, 2_000_001, B, 590_287_104, 546_151_168, 72_000_512),
    (True, 2_000_001, T | Q, 590_287_104, 722_160_896, 72_000_512),
    (True, 2_000_001, T | W4, 776_001_792, 722_160_896, 72_000_512),
]


@pytest.mark.parametrize("top, n, flags, structure, build, update", SIZES)
def test_sizes(rtlib, top, n, flags, structure, build, update):
    s = abi.RtBuildSizes()
    if top:
        assert rtlib.rt_get_tlas_build_sizes(n, flags, C.byref(s)) == abi.RT_OK
    else:
        g = (abi.RtGeometryTriangles * 1)()
        g[0].vertex_address, g[0].index_address, g[0].vertex_stride = 4096, 8192, 12
        g[0].max_vertex, g[0].primitive_count = 3 * n, n
        assert rtlib.rt_get_blas_build_sizes(g, 1, flags, C.byref(s)) == abi.RT_OK
    assert (s.acceleration_structure_size, s.build_scratch_size, s.update_scratch_size) == (structure, build, update)
