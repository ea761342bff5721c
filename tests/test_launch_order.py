"""Every kernel waits for the one before it.

All kernels are launched with programmatic dependent launch, so a kernel that
touches memory before its wait races with the previous kernel of its stream,
and one that ends without waiting lets the next kernel pass both.
"""

import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "ray-tracing-gallery_gb300" / "csrc"
KERNEL = re.compile(r"__global__[^;{]*?\b(k_[a-z0-9_]+)\s*\([^{;]*\)\s*\{\s*([^;]*);", re.S)


@pytest.mark.parametrize("source", ["rt_build.cu", "rt_trace.cu"])
def test_kernels_begin_with_the_wait(source):
    text = (CSRC / source).read_text()
    kernels = KERNEL.findall(text)
    assert len(kernels) == text.count("__global__")
    late = [name for name, first in kernels if not first.startswith("after_previous")]
    assert not late
