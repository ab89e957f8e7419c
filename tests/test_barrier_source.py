"""The grid barrier's accesses in the source.  What orders the phases before and after a barrier is a
release on arrival and an acquire on the poll, and the PTX memory model gives that only to accesses
that overlap completely.  No run on a GPU can show a violation, so the widths are read from the code:
arrival and poll are both 64 bits wide, and no kernel that uses the barrier reaches the error word,
the upper half of that word, with any other width."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "elmerfem_b200", "csrc")


def _read(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _body(src, start):
    i = src.index("{", src.index(start))
    depth = 0
    for j in range(i, len(src)):
        depth += {"{": 1, "}": -1}.get(src[j], 0)
        if depth == 0:
            return src[i:j]
    raise AssertionError(start)


def test_arrival_and_poll_have_one_width():
    src = _read("egpu_internal.cuh")
    body = _body(src, "bool grid_barrier(")
    calls = set(re.findall(r"\b((?:red|ld|st|atomic)\w*)\s*\(", body))
    assert calls, body
    widths = set()
    for c in calls:
        ptx = re.findall(r'"(?:red|ld|st|atom)[\w.]*\.(u|s|b)(\d+)', _body(src, c + "("))
        assert ptx, c
        widths |= {int(w) for _, w in ptx}
    assert widths == {64}


def test_error_word_is_reached_through_the_pair():
    """In every file whose kernels use the barrier, directly or through what they include."""
    files = [f for f in sorted(os.listdir(CSRC)) if f.endswith((".cu", ".cuh")) and f != "egpu_assembly.cu"]
    users = [f for f in files if "grid_barrier(" in _read(f)]
    assert {"egpu_internal.cuh", "egpu_krylov.cuh", "egpu_batch.cu", "egpu_noalloc.cu", "egpu_core.cu"} <= set(users)
    for f in files:
        src = _read(f)
        assert not re.search(r"atomic\w+\(\s*(?:\w+\.)?err\b", src), f
        assert not re.search(r"volatile int \*\)\s*(?:\w+\.)?err\b", src), f
