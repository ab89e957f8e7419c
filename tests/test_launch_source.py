"""The shared-memory limit of a kernel in the source: it belongs to the kernel on the device and not to
a context, so it is set in one place, to what a block can have at most, and never to the size of one
launch (a thread that lowers it between another thread's setting and launch has that launch
refused; the window is too short for a run to hit it reliably)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "elmerfem_b200", "csrc")


def test_shared_memory_limit_is_set_to_the_device_maximum_only():
    found = []
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh", ".h", ".cpp")):
            continue
        with open(os.path.join(CSRC, name)) as f:
            src = re.sub(r"//[^\n]*", "", f.read())
        found += [(name, src, m.start()) for m in re.finditer(r"cudaFuncSetAttribute\(", src)]
    assert len(found) == 1, [f[0] for f in found]
    _, src, at = found[0]
    start = src.rindex("int allow_shared(egpu_ctx *ctx, const void *kernel) {", 0, at)
    body = src[start:src.index("\n}", at)]
    assert "cudaDevAttrMaxSharedMemoryPerBlockOptin" in body and "sharedSizeBytes" in body
    assert "smem" not in body


def test_loading_a_kernel_is_asked_for_by_an_argument():
    """A launch whose arguments are not set fails or runs; it is never taken for a request to load only."""
    with open(os.path.join(CSRC, "egpu_krylov_launch.cuh")) as f:
        src = re.sub(r"//[^\n]*", "", f.read())
    body = src[src.index("int launch_coop("):]
    body = body[:body.index("\n}")]
    assert "load" in body and "args." not in body
    assert "cudaOccupancy" not in src  # asked once per context (kernel_blocks)
