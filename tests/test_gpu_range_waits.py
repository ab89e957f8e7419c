"""The row-range triangular solves after an error (needs a B200): the waits of a block for its staged
level records and for other blocks' values end by the context's limit, a cancelled solve leaves
in the middle of a triangle, no record is read before its copy is there, and the context and the
matrix stay usable.  Nothing here faults: each wait is bounded and the host reads a status."""
import threading
import time

import numpy as np
import pytest

import elmerfem_b200 as eg
import oracle
from elmerfem_b200 import _lib, meshgen
from helpers import elastic_problem, poisson_problem, rel, renumbered

pytestmark = pytest.mark.gpu

CASES = {
    "hex10": lambda: poisson_problem(meshgen.hex_cube(10))[::3],
    "hex32": lambda: poisson_problem(meshgen.hex_cube(32))[::3],
    "tet9_renumbered": lambda: poisson_problem(renumbered(meshgen.tet_cube(9), 3))[::3],
    "elastic8": lambda: elastic_problem(meshgen.hex_cube(8))[::3],  # node blocks
}


def _matrix(ctx, monkeypatch, p, v):
    monkeypatch.setenv("EGPU_TRI_MODE", "range")
    if p.dofs > 1:
        monkeypatch.setenv("EGPU_TRI_NODE_BLOCKS", "1")
    return eg.Matrix(ctx, eg.CRSPattern(p.n, p.nnz, p.dofs, p.perm, p.rows, p.cols, p.diag), v)


@pytest.mark.parametrize("limit", [2e-9, 5e-6])
@pytest.mark.parametrize("name", list(CASES))
def test_waits_run_out(ctx, monkeypatch, name, limit):
    """2 ns: a wait for a stage that is not over at its first look (the hardware's own wait of one
    try) is given up.  5 us: longer than a copy and shorter than a long chain of blocks, so it is
    values that are given up.  A solve in which no wait is that long has the right result."""
    p, v = CASES[name]()
    A = _matrix(ctx, monkeypatch, p, v)
    vs = v.copy()
    oracle.scale(p, vs)
    ilu, _ = A.ilu0(scale_system=True)
    b = np.random.default_rng(3).standard_normal(p.n)
    ref = oracle.lusolve(p, oracle.ilu0(p, vs), b)
    assert rel(A.lu_precondition(b), ref) < 1e-13
    for _ in range(3):
        ctx.set_wait_limit(limit)
        try:
            t0 = time.perf_counter()
            try:
                u = A.lu_precondition(b)
                assert name != "hex32" and rel(u, ref) < 1e-13  # hex32: 148 blocks in a chain, 90 us
            except _lib.LibError as e:
                assert e.code == -4  # EGPU_ERR_TIMEOUT
            assert time.perf_counter() - t0 < 1.0
        finally:
            ctx.set_wait_limit(0.0)
        assert rel(A.lu_precondition(b), ref) < 1e-13
    A.free()


@pytest.mark.parametrize("name", ["hex32", "elastic8"])
def test_cancelled_solve(ctx, monkeypatch, name):
    """A solve that would run for many seconds is cancelled from another thread; afterwards the
    same matrix solves correctly."""
    p, _, _, v, b, _ = elastic_problem(meshgen.hex_cube(8)) if name == "elastic8" else poisson_problem(meshgen.hex_cube(32))
    A = _matrix(ctx, monkeypatch, p, v)
    kw = dict(method=eg.BICGSTAB, precond=eg.PREC_ILU0)
    out = {}

    def run():
        # tolerance 1e-300: iterates until breakdown, so it is started again until cancelled
        try:
            end = time.perf_counter() + 30.0
            while time.perf_counter() < end:
                A.solve(b, params=eg.SolverParams(max_iter=1000000, tol=1e-300, abort_not_converged=False, **kw))
            out["rc"] = "not cancelled"
        except _lib.LibError as e:
            out["rc"] = e.code

    try:
        for _ in range(5):
            out.clear()
            th = threading.Thread(target=run)
            th.start()
            time.sleep(0.3)
            t0 = time.perf_counter()
            ctx.abort(True)
            th.join(timeout=60)
            assert not th.is_alive()
            assert out["rc"] == -7, out  # EGPU_ERR_ABORT
            assert time.perf_counter() - t0 < 2.0
            ctx.abort(False)
        x, r = A.solve(b, params=eg.SolverParams(max_iter=3000, tol=1e-10, **kw))
        x_ref, _ = oracle.solve(p, v, b, method=eg.BICGSTAB, precond=eg.PREC_ILU0, max_iter=3000, tol=1e-10)
        assert r["info"] == 1 and rel(x, x_ref) < 1e-8
    finally:
        ctx.abort(False)
        A.free()
