"""Acceleration-structure builds at the sizes where the builder changes path:
the one-block and grid-wide sorts, one clustering tile and several, the
one-CTA tail, single-leaf structures.  The blob is walked on the host (every
primitive in exactly one leaf, every node reached once, boxes nested) and rays
through it give the oracle's hits bit for bit."""
import numpy as np
import pytest

from oracle import oracle as O
from rtgallery import abi, scenes

pytestmark = pytest.mark.gpu

TRACE, BUILD = abi.RT_BUILD_PREFER_FAST_TRACE, abi.RT_BUILD_PREFER_FAST_BUILD
Q, W4 = abi.RT_BUILD_QUANTIZED_NODES, abi.RT_BUILD_EXT_NODE_WIDTH_4
EMPTY, LEAF = 0xFFFFFFFF, 0x80000000


def _host():
    from rtgallery import host

    return host


def _soup(n, kind, seed=5):
    rng = np.random.default_rng(seed + n)
    if kind == "same":        # one triangle n times: every area and key ties
        v = np.tile(rng.normal(size=(1, 3, 3)), (n, 1, 1))
    elif kind == "fan":       # slivers around one apex, as at the pole of a sphere
        a = np.arange(n + 1) * (2 * np.pi / n)
        ring = np.stack([np.cos(a), 0.05 * np.sin(3 * a), np.sin(a)], -1)
        v = np.stack([np.tile([[0.0, 0.3, 0.0]], (n, 1)), ring[:-1], ring[1:]], 1)
    else:                     # scattered small triangles
        v = rng.uniform(-3, 3, (n, 1, 3)) + rng.normal(scale=0.3, size=(n, 3, 3))
    pos = v.reshape(-1, 3).astype(np.float32)
    idx = np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)
    return scenes.Model(pos, np.zeros_like(pos), np.zeros((len(pos), 2), np.float32), [scenes.Geometry(idx)], kind)


def _scene(model, transforms):
    base = scenes.scene_small(8, 8)
    n = len(transforms)
    inst = scenes.instance_records(transforms, np.zeros(n), np.zeros(n), 0)
    return scenes.Scene([model], base.textures, inst, base.uniforms, 8, 8)


def _walk(acc, info, count, leaf_max):
    """Nodes of an FP32 blob: every primitive in one leaf, every node once, child boxes inside the parent's."""
    blob = acc.buffer.cpu().numpy()
    nodes = blob[512:512 + info.node_count * 256].view(np.float32).reshape(-1, 64)
    lo = np.stack([nodes[:, 0:8], nodes[:, 16:24], nodes[:, 32:40]], -1)
    hi = np.stack([nodes[:, 8:16], nodes[:, 24:32], nodes[:, 40:48]], -1)
    refs = nodes[:, 48:56].view(np.uint32)
    seen = np.zeros(count, np.int32)
    reached = np.zeros(info.node_count, np.int32)
    todo, depth = [(0, None, None)], 0
    while todo:
        depth += 1
        below = []
        for node, plo, phi in todo:
            reached[node] += 1
            for k in range(8):
                r = int(refs[node, k])
                if r == EMPTY:
                    continue
                if plo is not None:
                    assert (lo[node, k] >= plo).all() and (hi[node, k] <= phi).all()
                if r & LEAF:
                    first, m = r & 0x0FFFFFFF, ((r >> 28) & 7) + 1
                    assert m <= leaf_max
                    seen[first:first + m] += 1
                else:
                    below.append((r, lo[node, k], hi[node, k]))
        todo = below
    assert (seen == 1).all() and (reached == 1).all() and depth == info.tree_depth


def _check(device, sc, blas_flags, tlas_flags, walk):
    host = _host()
    gs = host.GpuScene(device, sc, blas_flags=blas_flags, tlas_flags=tlas_flags)
    rays = scenes.random_rays(3000, 17, 8.0)
    rays["tmax"] = 1e4
    device.read_stats(reset=True)
    g = host.trace_ray_buffer(device, gs, rays, with_models=False)
    assert device.read_stats(reset=True)["status"] == 0
    o, _ = O.OracleScene(sc).trace(rays, with_models=False)
    for f in ("t", "u", "v", "instance_id", "geometry_index", "primitive_index", "hit_kind"):
        assert (np.asarray(g[f]).view(np.uint32) == np.asarray(o[f]).view(np.uint32)).all(), f
    for acc, n, leaf in ((gs.models[0].blas, sc.models[0].triangle_count, 2), (gs.tlas, len(sc.instances), 1)):
        info = acc.info(device)
        assert info.status == 0 and info.primitive_count == n
        if walk and info.node_bytes == 256:
            _walk(acc, info, n, leaf)


BLAS_SIZES = [1, 2, 3, 9, 31, 33, 448, 1023, 1024, 1025, 2049, 4097, 8193, 16385, 20011]


@pytest.mark.parametrize("n", BLAS_SIZES)
@pytest.mark.parametrize("flags", [TRACE, BUILD, TRACE | Q, TRACE | W4, BUILD | Q], ids=["ploc", "karras", "ploc_q8",
                                                                                         "ploc_w4", "karras_q8"])
def test_blas_sizes(device, n, flags):
    _check(device, _scene(_soup(n, "soup"), scenes.affine(np.eye(3), [0, 0, 0])[None]), flags,
           TRACE | abi.RT_BUILD_ALLOW_UPDATE, walk=True)


@pytest.mark.parametrize("n", [5, 1024, 1500, 9000])
@pytest.mark.parametrize("kind", ["same", "fan"])
@pytest.mark.parametrize("flags", [TRACE, BUILD], ids=["ploc", "karras"])
def test_blas_of_ties_and_slivers(device, n, kind, flags):
    _check(device, _scene(_soup(n, kind), scenes.affine(np.eye(3), [0, 0, 0])[None]), flags,
           TRACE | abi.RT_BUILD_ALLOW_UPDATE, walk=True)


@pytest.mark.parametrize("n", [1, 2, 8, 9, 31, 33, 127, 256, 257, 1023, 1024, 1025, 2048, 2049, 4500])
@pytest.mark.parametrize("flags", [TRACE, BUILD, TRACE | W4], ids=["ploc", "karras", "ploc_w4"])
def test_tlas_sizes(device, n, flags):
    rng = np.random.default_rng(n)
    xf = np.stack([scenes.affine(scenes.rot_y(rng.uniform(0, 6)), rng.uniform(-4, 4, 3), rng.uniform(0.05, 0.4))
                   for _ in range(n)])
    xf[n // 2] = 0.0  # a singular transform among them: never hit
    _check(device, _scene(_soup(12, "soup"), xf), TRACE, flags | abi.RT_BUILD_ALLOW_UPDATE, walk=False)


@pytest.mark.parametrize("n", [1, 2, 9, 65, 511, 512, 513, 1500])
@pytest.mark.parametrize("flags", [TRACE, TRACE | W4], ids=["w8", "w4"])
def test_tlas_refit_sizes(device, n, flags):
    """Every instance moved and the TLAS refitted in place: the hits of the oracle's fresh structure."""
    host = _host()
    rng = np.random.default_rng(n)

    def transforms():
        return np.stack([scenes.affine(scenes.rot_y(rng.uniform(0, 6)), rng.uniform(-4, 4, 3), rng.uniform(0.05, 0.4))
                         for _ in range(n)])

    model = _soup(12, "soup")
    gs = host.GpuScene(device, _scene(model, transforms()), tlas_flags=flags | abi.RT_BUILD_ALLOW_UPDATE)
    moved = _scene(model, transforms())
    instances = host.Device.upload(gs.patch_instances(moved.instances))
    gs.tlas.update_tlas(device, instances, n, gs.scratch)
    rays = scenes.random_rays(3000, 23, 8.0)
    rays["tmax"] = 1e4
    g = host.trace_ray_buffer(device, gs, rays, with_models=False)
    o, _ = O.OracleScene(moved).trace(rays, with_models=False)
    for f in ("t", "u", "v", "instance_id", "primitive_index"):
        assert (np.asarray(g[f]).view(np.uint32) == np.asarray(o[f]).view(np.uint32)).all(), f
    assert gs.tlas.info(device).status == 0
