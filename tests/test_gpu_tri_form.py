"""Which form the triangular solves take (egpu_tri_form): that the cases of test_gpu_tri_range.py run in
row ranges, for both widths of a lane, that a plan which fits shared memory in FP32 only is used
there and nowhere else, and that ILUT's factor runs in row ranges where that is asked for."""
import numpy as np
import pytest

import elmerfem_b200 as eg
import oracle
from elmerfem_b200 import meshgen
from helpers import elastic_problem, poisson_problem, rel
from test_gpu_tri_range import CASES, _matrix

pytestmark = pytest.mark.gpu

SHAPES = {  # lanes and entries a lane, from the longest triangle row: 13, 39 and 39 entries
    "hex10": (2, 7), "hex32": (2, 7), "elastic8": (4, 10),
}


@pytest.mark.parametrize("ranges", [3, 148])
@pytest.mark.parametrize("name", list(CASES))
def test_lu_precondition_cases(ctx, monkeypatch, name, ranges):
    p, v = CASES[name]()
    A = _matrix(ctx, monkeypatch, p, v, ranges)
    A.ilu0(scale_system=True)
    form = A.tri_form()
    if (name, ranges) == ("hex32", 3):  # 11,979 rows a range: 274 KB in FP64
        assert form["form"] != "ranges"
        return
    bs = A.tri_info()["node_block"]  # a whole number of node blocks a range
    per = -(-(-(-p.n // ranges)) // bs) * bs
    assert form["form"] == "ranges" and form["ranges"] == -(-p.n // per)
    if name in SHAPES:
        assert (form["lanes"], form["entries"]) == SHAPES[name]
    A.free()


@pytest.mark.parametrize("name", ["hex10", "hex32", "elastic8"])
def test_solve_cases(ctx, monkeypatch, name):
    p, v = CASES[name]()
    A = _matrix(ctx, monkeypatch, p, v, 20)
    A.ilu0(scale_system=True)
    for precision in (eg.FP64, eg.MIXED):
        form = A.tri_form(precision)
        assert form["form"] == "ranges" and form["ranges"] == 20
        assert (form["lanes"], form["entries"]) == SHAPES[name]
    A.free()


def test_wide_ranges_apply(ctx, monkeypatch):
    """Six ranges of hex32: the widest that fit in FP64."""
    p, v = CASES["hex32"]()
    A = _matrix(ctx, monkeypatch, p, v, 6)
    ilu, _ = A.ilu0(scale_system=True)
    assert A.tri_form()["form"] == "ranges" and A.tri_form()["ranges"] == 6
    b = np.random.default_rng(3).standard_normal(p.n)
    assert rel(A.lu_precondition(b), oracle.lusolve(p, ilu, b)) < 1e-13
    A.free()


@pytest.mark.parametrize("method", [eg.CG, eg.BICGSTAB], ids=["cg", "bicgstab"])
def test_fp32_only_plan(ctx, monkeypatch, method):
    """Three ranges of hex32 fit in FP32 only: the mixed solve's inner solves take them, an FP64 solve
    of the same matrix another form."""
    monkeypatch.setenv("EGPU_MIXED_AUTO", "0")
    p, _, _, v, b, _ = poisson_problem(meshgen.hex_cube(32))
    A = _matrix(ctx, monkeypatch, p, v, 3)
    A.ilu0(scale_system=True)
    assert A.tri_form(eg.FP64)["form"] != "ranges"
    assert A.tri_form(eg.MIXED)["form"] == "ranges" and A.tri_form(eg.MIXED)["ranges"] == 3
    x_ref, r_ref = oracle.solve(p, v, b, method=method, precond=eg.PREC_ILU0, max_iter=3000, tol=1e-12)
    for precision in (eg.MIXED, eg.FP64):
        x, r = A.solve(b, params=eg.SolverParams(method=method, precond=eg.PREC_ILU0, max_iter=3000, tol=1e-12,
                                                 precision=precision, ilu_sweeps=0))
        assert r["info"] == 1 and r["precision_used"] == precision
        assert rel(x, x_ref) < 1e-8
    A.free()


@pytest.mark.parametrize("order", [1, 2])
def test_ilun_shape(ctx, monkeypatch, order):
    """The shape with the fewest entries that holds the longest triangle row of ILU(n)."""
    p, _, _, v, b, _ = poisson_problem(meshgen.hex_cube(8))
    A = _matrix(ctx, monkeypatch, p, v, 20)
    A.solve(b, params=eg.SolverParams(method=eg.BICGSTAB, precond=eg.PREC_ILU0, max_iter=1000, tol=1e-10, ilu_order=order))
    r, _, d, _ = A.ilu_factors()
    entries = max(np.max(d - r[:-1]), np.max(r[1:] - d - 1))
    fits = [(g * k, g, k) for g in (1, 2, 4, 8) for k in (7, 10) if g * k >= entries]
    form = A.tri_form()
    assert (form["form"] == "ranges") == bool(fits)
    if fits:
        assert (form["lanes"], form["entries"]) == min(fits)[1:]
    A.free()


@pytest.mark.parametrize("name,tol", [("hex10", 1e-3), ("hex10", 0.0), ("elastic4", 1e-3)])
def test_ilut_in_ranges(ctx, monkeypatch, name, tol):
    p, v = CASES["hex10"]() if name == "hex10" else elastic_problem(meshgen.hex_cube(4))[::3]
    A = _matrix(ctx, monkeypatch, p, v, 20)
    r, c, d, val = A.ilut(tol)
    entries = max(np.max(d - r[:-1]), np.max(r[1:] - d - 1))
    assert (A.tri_form()["form"] == "ranges") == bool(entries <= 80)  # eight lanes of ten entries
    b = np.random.default_rng(4).standard_normal(p.n)
    assert rel(A.lu_precondition(b), oracle.lusolve_on(r, c, d, val, b)) < 1e-13
    A.free()
