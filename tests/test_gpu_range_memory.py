"""Triangular solves where the row ranges' buffers do not fit the free device memory: the solve takes another
form, as it did before the ranges were offered, and reports no error."""
import numpy as np
import pytest
import torch

import elmerfem_b200 as eg
import oracle
from elmerfem_b200 import meshgen
from helpers import poisson_problem, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("left_mb", [40, 6], ids=["records", "plan"])
def test_other_form_without_memory(monkeypatch, left_mb):
    """hex 64^3: plan 28 MB, FP64 level records 39 MB a triangle."""
    p, _, _, v, b, _ = poisson_problem(meshgen.hex_cube(64))
    ctx = eg.Context(0)
    A = eg.Matrix(ctx, eg.CRSPattern(p.n, p.nnz, 1, p.perm, p.rows, p.cols, p.diag), v)
    monkeypatch.setenv("EGPU_TRI_MODE", "syncfree")
    ilu, _ = A.ilu0()
    ref = oracle.lusolve(p, ilu, b)
    assert rel(A.lu_precondition(b), ref) < 1e-13  # every other buffer is allocated now
    prm = eg.SolverParams(method=eg.BICGSTAB, precond=eg.PREC_ILU0, max_iter=500, tol=1e-10)
    x_ref, r_ref = A.solve(b, params=prm)
    monkeypatch.delenv("EGPU_TRI_MODE")
    eg.release_cached_memory()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    filler = torch.empty(free - (left_mb << 20), dtype=torch.uint8, device="cuda")
    try:
        assert torch.cuda.mem_get_info()[0] < (left_mb + 8) << 20
        assert rel(A.lu_precondition(b), ref) < 1e-13
        assert A.tri_form()["form"] != "ranges"
        x, r = A.solve(b, params=prm)
        assert r["info"] == 1 and r["iters"] == r_ref["iters"] and np.array_equal(x, x_ref)
    finally:
        del filler
        torch.cuda.empty_cache()
    A.free()
    ctx.close()
