"""Climbs from the leaves up: the last to arrive at a node reads what the others wrote.

An arrival must order the climbing thread's own box before it and its reads of
the other children's boxes after it.  A relaxed atomic with a fence before it
does the first only; a box read too early would be smaller than its child.
"""
import pathlib
import re

import pytest

SOURCE = pathlib.Path(__file__).resolve().parent.parent / "ray-tracing-gallery_gb300" / "csrc" / "rt_build.cu"


def _kernel(name):
    text = re.sub(r"//[^\n]*", "", SOURCE.read_text())
    found = re.search(r"__global__[^;{]*?\b%s\s*\([^{;]*\)\s*(\{.*?\n\})" % name, text, re.S)
    return found.group(1)


@pytest.mark.parametrize("name", ["k_bottom_up", "k_refit_nodes"])
def test_grid_wide_arrivals_acquire_and_release(name):
    body = _kernel(name)
    assert len(re.findall(r"\barrive\(", body)) == 1
    assert "atomicAdd" not in body
    helper = re.search(r"uint32_t arrive\(uint32_t\* \w+\) \{(.*?)\n\}", SOURCE.read_text(), re.S).group(1)
    assert "atom.acq_rel.gpu.global.add.u32" in helper and '"memory"' in helper


def test_one_block_arrivals_are_fenced_for_the_whole_group():
    body = _kernel("k_refit_small")
    order = [r"__threadfence_block\(\);", r"atomicAdd\(&arrived\[", r"__threadfence_block\(\);", r"last = __shfl_sync",
             r"__syncwarp\(gmask\);"]
    assert re.search(".*?".join(order), body, re.S)
