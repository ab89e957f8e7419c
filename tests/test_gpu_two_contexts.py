"""Two contexts, a thread each, on one GPU: kernels with different amounts of shared memory.  What a
launch may use is an attribute of the kernel on the device and not of a context, so no context may
lower it under another one's launch."""
import threading

import numpy as np
import pytest

import elmerfem_b200 as eg
import oracle
from elmerfem_b200 import meshgen
from helpers import poisson_problem, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["range", "block"])
def test_triangular_solves_of_two_sizes(monkeypatch, mode):
    monkeypatch.setenv("EGPU_TRI_MODE", mode)
    work = []
    # range: one and two ranges, about 110 and 80 KB a block; block: rings of two sizes.  Each twice
    for cells, ranges in 2 * (((12, 1), (12, 2)) if mode == "range" else ((16, 0), (10, 0))):
        monkeypatch.setenv("EGPU_TRI_RANGES", str(ranges))
        p, _, _, v, _, _ = poisson_problem(meshgen.hex_cube(cells))
        ctx = eg.Context(0)
        A = eg.Matrix(ctx, eg.CRSPattern(p.n, p.nnz, 1, p.perm, p.rows, p.cols, p.diag), v)
        ilu, _ = A.ilu0(scale_system=True)
        b = np.random.default_rng(cells).standard_normal(p.n)
        ref = oracle.lusolve(p, ilu, b)
        assert rel(A.lu_precondition(b), ref) < 1e-13
        work.append((ctx, A, b, ref))
    failed = []

    def run(A, b, ref):
        try:
            for _ in range(5000):
                u = A.lu_precondition(b)
            assert rel(u, ref) < 1e-13
        except Exception as e:  # noqa: BLE001
            failed.append(repr(e))

    threads = [threading.Thread(target=run, args=w[1:]) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=120)
    for ctx, A, _, _ in work:
        A.free()
        ctx.close()
    assert not failed
