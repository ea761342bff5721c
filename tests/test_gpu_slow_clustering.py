"""Meshes whose clusters merge more slowly than the grid-wide rounds count on.

Nested shells: in a stack of boxes, each around the last, every box's nearest
neighbour is one further in, so one pair of a stack merges in a round and the
rounds that are launched leave more clusters than the last block takes.  The
rest is merged in neighbour pairs; the structure is walked and its hits are the
oracle's.
"""
import math

import numpy as np
import pytest

from rtgallery import abi, scenes
from test_gpu_build_edges import TRACE, W4, Q, _check, _scene

SHELLS, RADIUS, TAIL = 30, 16, 1024


def _rounds(n):
    """Grid-wide clustering rounds of a build of n primitives (more than the tail takes)."""
    x = 0.62 * n / TAIL
    return 1 + (math.ceil(math.log(x) / -math.log(0.765)) if x > 1 else 0) + 6


def _round(areas, first):
    """One round over a stack alone: areas[i] = the area of cluster i, which holds all before it."""
    n = len(areas)
    if n < 2:
        return areas

    def merged(i, j):
        return areas[max(i, j)]

    near = [min((merged(i, j), j) for j in range(max(0, i - RADIUS), min(n, i + RADIUS + 1)) if j != i)[1]
            for i in range(n)]
    mutual = [near[near[i]] == i for i in range(n)]
    takes = {}
    for i in range(n):
        j = near[i]
        if not mutual[i] and not mutual[j] and (first + i) % 2 and not (first + j) % 2:
            if merged(i, j) <= merged(j, near[j]) * 1.25:
                takes[j] = min(takes.get(j, (math.inf, 0)), (merged(i, j), i))
    pairs = [(i, near[i]) for i in range(n) if mutual[i]] + [(i, j) for j, (_, i) in takes.items()]
    gone = {max(p) for p in pairs}
    grown = {min(p): merged(*p) for p in pairs}
    return [grown.get(i, areas[i]) for i in range(n) if i not in gone]


def _left(rounds):
    """The most that the rounds take from a stack, whatever the parity of its first place."""
    fewest = [list(1.1 ** (2 * np.arange(SHELLS)))]
    for _ in range(rounds):
        fewest = [min((_round(a, first) for first in (0, 1)), key=len) for a in fewest]
    return len(fewest[0])


def _shells(stacks):
    rng = np.random.default_rng(stacks)
    side = math.ceil(stacks ** (1 / 3))
    cells = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:stacks]
    centre = (cells + rng.uniform(0.4, 0.6, (stacks, 3))) * (6.0 / side) - 3.0
    size = 0.005 * 1.1 ** np.arange(SHELLS)
    corners = np.array([[-1, -1, -1], [1, 1, -1], [-1, 1, 1]], np.float64)  # its box is the cube
    v = centre[:, None, None, :] + size[None, :, None, None] * corners[None, None]
    pos = v.reshape(-1, 3).astype(np.float32)
    idx = np.arange(len(pos), dtype=np.uint32).reshape(-1, 3)
    return scenes.Model(pos, np.zeros_like(pos), np.zeros((len(pos), 2), np.float32), [scenes.Geometry(idx)], "shells")


@pytest.mark.parametrize("stacks", [46, 64, 200, 4096])
def test_the_rounds_leave_too_many(stacks):
    assert stacks * _left(_rounds(stacks * SHELLS)) > TAIL


@pytest.mark.gpu
@pytest.mark.parametrize("stacks", [46, 64, 200, 4096])
@pytest.mark.parametrize("flags", [TRACE, TRACE | W4, TRACE | Q], ids=["w8", "w4", "q8"])
def test_nested_shells(device, stacks, flags):
    _check(device, _scene(_shells(stacks), scenes.affine(np.eye(3), [0, 0, 0])[None]), flags,
           TRACE | abi.RT_BUILD_ALLOW_UPDATE, walk=True)
