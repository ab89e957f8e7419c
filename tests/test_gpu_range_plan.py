"""When the row ranges of the triangular solves are planned: by the preparation or the first exact solve
of a precision that they can serve, and by nothing else.  The plan's two index kernels show in the launch count."""
import pytest

import elmerfem_b200 as eg
import oracle
from elmerfem_b200 import _lib, meshgen
from helpers import poisson_problem, rel

pytestmark = pytest.mark.gpu


def _matrix(ctx, cells=16):
    p, _, _, v, b, _ = poisson_problem(meshgen.hex_cube(cells))
    return p, v, b, eg.Matrix(ctx, eg.CRSPattern(p.n, p.nnz, p.dofs, p.perm, p.rows, p.cols, p.diag), v)


def _launches(ctx):
    return int(_lib.lib().egpu_kernel_launches(ctx.handle))


@pytest.fixture(autouse=True)
def _default_forms(monkeypatch):
    for name in ("EGPU_TRI_MODE", "EGPU_TRI_RANGES", "EGPU_ILU_SWEEPS"):
        monkeypatch.delenv(name, raising=False)
    monkeypatch.setenv("EGPU_MIXED_AUTO", "0")


def test_preparation_for_exact_solves_plans(ctx):
    """After it, the first solve on a pattern costs what later ones do."""
    for prm in (dict(), dict(precision=eg.MIXED, ilu_sweeps=0), dict(precision=eg.MIXED)):
        p, v, b, A = _matrix(ctx)
        n0 = _launches(ctx)
        A.prepare(eg.SolverParams(method=eg.BICGSTAB, precond=eg.PREC_ILU0, **prm))
        assert _launches(ctx) - n0 == 2
        A.ilu0()
        n0 = _launches(ctx)
        assert A.tri_form(prm.get("precision", eg.FP64))["form"] == "ranges"
        assert _launches(ctx) == n0
        A.free()


def test_factorisation_plans_nothing(ctx):
    p, v, b, A = _matrix(ctx)
    n0 = _launches(ctx)
    A.prepare(eg.SolverParams(method=eg.BICGSTAB, precond=eg.PREC_ILU0, precision=eg.MIXED, ilu_sweeps=2))
    assert _launches(ctx) == n0
    ilu, _ = A.ilu0()
    n1 = _launches(ctx)
    assert A.tri_form()["form"] == "ranges"
    n2 = _launches(ctx)
    assert n2 - n1 == 2  # one index kernel a triangle, now
    A.ilu0()
    assert _launches(ctx) - n2 == n1 - n0  # and not again
    x = A.lu_precondition(b)
    assert rel(x, oracle.lusolve(p, ilu, b)) < 1e-13
    A.free()


def test_sweeps_plan_nothing(ctx):
    p, v, b, A = _matrix(ctx)
    x, r = A.solve(b, params=eg.SolverParams(method=eg.BICGSTAB, precond=eg.PREC_ILU0, max_iter=500, tol=1e-10,
                                             precision=eg.MIXED, ilu_sweeps=2))
    assert r["ilu_sweeps_used"] == 2
    n0 = _launches(ctx)
    assert A.tri_form(eg.MIXED)["form"] == "ranges"
    assert _launches(ctx) - n0 == 2
    A.free()


def test_ilut_is_not_planned_unasked(ctx):
    p, v, b, A = _matrix(ctx, 10)
    for _ in range(2):
        r, c, d, val = A.ilut(1e-3)
        n0 = _launches(ctx)
        assert A.tri_form()["form"] != "ranges"
        assert _launches(ctx) == n0
        assert rel(A.lu_precondition(b), oracle.lusolve_on(r, c, d, val, b)) < 1e-13
    A.free()


def test_clones_share_one_plan(ctx):
    p, v, b, A = _matrix(ctx)
    ref = oracle.lusolve(p, A.ilu0()[0], b)
    B = eg.Matrix.clone(A)
    C = eg.Matrix.clone(A)
    B.update_values(v)
    C.update_values(4.0 * v)
    for M in (B, C):
        M.ilu0()  # scaled to a unit diagonal, powers of two: the same factor
    n0 = _launches(ctx)
    assert B.tri_form()["form"] == "ranges"
    assert _launches(ctx) - n0 == 2
    assert C.tri_form() == B.tri_form() and A.tri_form() == B.tri_form()
    assert _launches(ctx) - n0 == 2
    for M in (A, B, C):
        assert rel(M.lu_precondition(b), ref) < 1e-13
    for M in (B, C, A):
        M.free()


def test_footprint_counts_the_level_records(ctx):
    """A solve in row ranges holds the level records of its precision: per row and padded entry an index of
    two bytes and a value of eight or four, in both triangles."""
    p, v, b, A = _matrix(ctx)
    A.ilu0()
    none = A.footprint(eg.PREC_NONE)
    before = A.footprint(eg.PREC_ILU0)
    form = A.tri_form()
    assert form["form"] == "ranges"
    extra = A.footprint(eg.PREC_ILU0) - before
    entries = 2 * p.n * form["lanes"] * form["entries"]
    least = entries * (10 + 6)
    assert least <= extra <= 1.3 * least  # row numbers, headers and padding besides
    assert A.footprint(eg.PREC_NONE) == none
    A.free()
