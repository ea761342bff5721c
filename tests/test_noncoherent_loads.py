"""No kernel reads through the non-coherent cache what may still be written.

A kernel launched with programmatic overlap is resident while the kernel before
it runs.  Non-coherent loads (ld.global.nc: __ldg, const __restrict__) are only
defined for data that nothing writes while the kernel is resident, and the
compiler may move them across the wait.  So a kernel that uses them is launched
without overlap, or behind kernels of its own sequence that write none of it.
"""
import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parent.parent / "ray-tracing-gallery_gb300" / "csrc"
NONCOHERENT = re.compile(r"__ldg|__restrict__|ld\.global\.nc")


def _code(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


def _body(text, head):
    """The braces that follow the definition `head`."""
    at = text.index("{", text.index(head))
    depth = 0
    for end in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        if depth == 0:
            return text[at:end]
    raise AssertionError(head)


def test_builder_kernels_use_none():
    assert not NONCOHERENT.search(_code("rt_build.cu"))


def test_ray_buffer_kernel_does_not_overlap():
    """It follows whatever the caller queued: a build, a refit, a copy, the kernel that made its rays."""
    launches = re.findall(r"launch(<false>)?\(k_trace_ray_buffer", _code("rt_trace.cu"))
    assert launches and all(launches)


def test_frames_put_two_kernels_before_the_traversal():
    """Setup and camera rays use none, and each waits for the kernel before it, so everything that was
    queued before the frame is complete when the first traversal becomes resident."""
    text = _code("rt_trace.cu")
    for source, head in ((text, "__global__ void k_setup("), (text, "__global__ void k_raygen("),
                         (_code("rt_shade.cuh"), "Env make_env(")):
        assert not NONCOHERENT.search(_body(source, head)), head
    order = _body(text, "cudaError_t launch_trace_batch(")
    places = [order.index(s) for s in ("launch(k_setup", "launch(k_raygen", "launch_trace_mode<kModeBounce>")]
    assert places == sorted(places)


def test_traversals_do_not_let_the_next_kernel_in_early():
    """Shading samples textures with them, and starts when the traversal before it has completed."""
    text = _code("rt_trace.cu")
    for kernel in ("k_trace", "k_trace_packet", "k_trace_ray_buffer"):
        body = _body(text, kernel + "(const __grid_constant__")
        assert "after_previous_alone();" in body and "after_previous();" not in body
