"""Copies in the source: in the order of the context's stream.  cudaMemcpy and cudaMemset belong to the
legacy stream, which the context's non-blocking stream does not wait for, and a copy from pageable
memory may return before the data is in place; a kernel launched next on the context's stream can
then read what the buffer held before (a plan's index lists: indices out of range).  Whether it
does depends on the machine's timing, so the calls are looked for in the code."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "elmerfem_b200", "csrc")


def test_no_legacy_stream_copies_beside_the_contexts_stream():
    seen = 0
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh", ".h", ".cpp")):
            continue
        if name == "egpu_noalloc.cu":  # no context: all its work is on the legacy stream
            continue
        with open(os.path.join(CSRC, name)) as f:
            src = re.sub(r"//[^\n]*", "", f.read())
        calls = re.findall(r"\bcudaMem(?:cpy|set)(?:2D|3D)?\s*\(", src)
        assert not calls, (name, calls)
        seen += len(re.findall(r"\b(?:egpu_copy|cudaMemcpyAsync|cudaMemsetAsync)\(", src))
    assert seen > 50
