"""Clustering chooses between neighbours by whole 32-bit areas.

Rows of three boxes A, B, C: merging B with C is smaller than merging it with A
by a few units in the last place, less than 2^-18 of the area.  B and C must be
the pair (ties alone go to the lower position, A)."""
import numpy as np
import pytest

from rtgallery import abi, scenes
from test_gpu_build_edges import EMPTY, LEAF, TRACE, _scene

F = np.float32


def _padded(lo, hi):
    pad = np.maximum(np.abs(lo), np.abs(hi)) * F(2.0 ** -20) + F(1e-30)
    return lo - pad, hi + pad


def _area(a, b):
    """Half the surface area of two padded boxes together, as the builder computes it in float."""
    e = np.maximum(a[1], b[1]) - np.minimum(a[0], b[0])
    return F(np.float64(e[0]) * np.float64(e[1] + e[2]) + np.float64(e[1] * e[2]))


def _rows(count):
    """`count` rows of three unit boxes along x, A taller than B and C by a few units in the last place."""
    rows, k = [], 0
    while len(rows) < count:
        x = F(8 * k + 1)
        k += 1
        boxes = []
        for j, height in enumerate((F(1) + F(1e-6), F(1), F(1))):
            boxes.append((np.array([x + F(j), 0, 0], F), np.array([x + F(j + 1), height, 1], F)))
        a, b, c = (_padded(*box) for box in boxes)
        ab, bc, ac = _area(a, b), _area(b, c), _area(a, c)
        near = (ab.view(np.uint32) & ~np.uint32(31)) == (bc.view(np.uint32) & ~np.uint32(31))
        if bc < ab < ac and near:
            rows.append(boxes)
    return rows


def _model(rows):
    lo = np.array([b[0] for r in rows for b in r], F)
    hi = np.array([b[1] for r in rows for b in r], F)
    v = np.stack([lo, np.stack([hi[:, 0], hi[:, 1], lo[:, 2]], -1), np.stack([lo[:, 0], hi[:, 1], hi[:, 2]], -1)], 1)
    pos = v.reshape(-1, 3)
    idx = np.arange(len(pos), dtype=np.uint32).reshape(-1, 3)
    return scenes.Model(pos, np.zeros_like(pos), np.zeros((len(pos), 2), F), [scenes.Geometry(idx)], "rows")


COUNTS = [1, 7, 300, 400]  # one block; the last one also grid-wide


@pytest.mark.parametrize("count", COUNTS)
def test_rows_are_as_described(count):
    rows = _rows(count)
    assert len(rows) == count and max(r[2][1][0] for r in rows) < 6000


@pytest.mark.gpu
@pytest.mark.parametrize("count", COUNTS)
def test_the_nearer_of_two_almost_equal_neighbours(device, count):
    from rtgallery import host

    gs = host.GpuScene(device, _scene(_model(_rows(count)), scenes.affine(np.eye(3), [0, 0, 0])[None]), blas_flags=TRACE,
                       tlas_flags=TRACE | abi.RT_BUILD_ALLOW_UPDATE)
    blas = gs.models[0].blas
    info = blas.info(device)
    blob = blas.buffer.cpu().numpy()
    refs = blob[512:512 + info.node_count * 256].view(np.uint32).reshape(-1, 64)[:, 48:56].reshape(-1)
    prims = blob[:64].view(np.uint64)[6]
    order = blob[prims:prims + 48 * 3 * count].view(np.uint32).reshape(-1, 12)[:, 3]
    pairs = set()
    for r in refs[(refs != EMPTY) & (refs & LEAF != 0)]:
        first, m = int(r) & 0x0FFFFFFF, ((int(r) >> 28) & 7) + 1
        if m == 2:
            pairs.add(tuple(sorted(int(p) for p in order[first:first + 2])))
    for row in range(count):
        assert (3 * row + 1, 3 * row + 2) in pairs, row
