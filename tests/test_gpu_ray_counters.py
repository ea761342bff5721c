"""Ray-buffer queries that overlap, and the calls that come after them.

A query longer than the lanes of its grid hands its rays out from a counter.
More queries than there once were counters are kept in flight on two streams,
and a captured query is replayed beside direct ones; every hit of every call,
then and afterwards, is the one that the query gives alone.
"""
import numpy as np
import pytest

from oracle import oracle as O
from rtgallery import scenes

pytestmark = pytest.mark.gpu

LONG, SHORT = 200_003, 1_000  # above and below the lanes of the grid (152 SMs of 24 or 32 warps)
CALLS = 300                   # per stream


class Query:
    def __init__(self, device):
        import torch

        from rtgallery import abi, host

        self.device, self.torch, self.size = device, torch, abi.HIT_DTYPE.itemsize
        scene = scenes.scene_gallery(8, 8)
        self.scene = host.GpuScene(device, scene)
        rays = scenes.random_rays(LONG, 41, 16.0)
        self.rays = host.Device.upload(rays)
        self.alone = self.hits(LONG)
        self.call(self.alone, torch.cuda.current_stream())
        torch.cuda.synchronize()
        got = self.alone.cpu().numpy().view(abi.HIT_DTYPE).reshape(-1)
        want, _ = O.OracleScene(scene).trace(rays, with_models=False)
        for f in ("t", "u", "v", "instance_id", "geometry_index", "primitive_index"):
            assert (np.asarray(got[f]).view(np.uint32) == np.asarray(want[f]).view(np.uint32)).all(), f

    def hits(self, count, calls=None):
        shape = (count * self.size,) if calls is None else (calls, count * self.size)
        return self.torch.zeros(shape, dtype=self.torch.uint8, device="cuda")

    def call(self, hits, stream):
        d = self.device
        d.check(d.lib.rt_cmd_trace_ray_buffer(d.ctx, self.scene.tlas.device_address(), None, None, 0, 0xFF, 0,
                                              self.rays.data_ptr(), hits.numel() // self.size, hits.data_ptr(),
                                              stream.cuda_stream))

    def check(self, rows):
        want = self.alone[: rows.shape[-1]]
        assert bool((rows.reshape(-1, rows.shape[-1]) == want).all())

    def check_single_calls(self):
        """One query after the other, over more calls than there once were counters."""
        rows = self.hits(LONG, CALLS)
        for row in rows:
            self.call(row, self.torch.cuda.current_stream())
        self.torch.cuda.synchronize()
        self.check(rows)


@pytest.fixture(scope="module")
def query(device):
    return Query(device)


@pytest.mark.parametrize("count", [SHORT, LONG])
def test_many_queries_on_two_streams(query, count):
    torch = query.torch
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    rows = [query.hits(count, CALLS) for _ in streams]
    torch.cuda.synchronize()
    for k in range(CALLS):
        for r, s in zip(rows, streams):
            query.call(r[k], s)
    torch.cuda.synchronize()
    for r in rows:
        query.check(r)
    query.check_single_calls()


def test_captured_query_beside_direct_ones(query):
    torch = query.torch
    replayed, side = torch.cuda.Stream(), torch.cuda.Stream()
    mine = query.hits(LONG)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=replayed):
        query.call(mine, torch.cuda.current_stream())
    rows, copies = query.hits(LONG, CALLS), query.hits(LONG, 60)
    torch.cuda.synchronize()
    for k in range(CALLS):
        query.call(rows[k], side)
        if k % 5 == 0:
            with torch.cuda.stream(replayed):
                mine.zero_()
                g.replay()
                copies[k // 5].copy_(mine)
    torch.cuda.synchronize()
    query.check(rows)
    query.check(copies)
    query.check_single_calls()
