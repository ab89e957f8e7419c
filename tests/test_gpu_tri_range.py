"""Row-range triangular solves (EGPU_TRI_MODE=range) against the oracle: rows and node blocks, one
range and many, 4 and 5 entries a lane, rows of ILU(1), FP64 and the FP32 inner solves."""
import numpy as np
import pytest

import elmerfem_b200 as eg
import oracle
from elmerfem_b200 import meshgen
from helpers import elastic_problem, poisson_problem, rel, renumbered

pytestmark = pytest.mark.gpu


def _dofs(mesh, dofs):
    p = oracle.create_pattern(mesh, dofs=dofs)
    v = np.random.default_rng(5).uniform(-1.0, 1.0, p.nnz)
    v[p.diag - 1] = np.diff(p.rows).astype(np.float64) + 1.0
    return p, v


def _poisson(mesh):
    t = poisson_problem(mesh)
    return t[0], t[3]


CASES = {
    "hex2": lambda: _poisson(meshgen.hex_cube(2)),
    "hex10": lambda: _poisson(meshgen.hex_cube(10)),
    "hex32": lambda: _poisson(meshgen.hex_cube(32)),
    "tet9_renumbered": lambda: _poisson(renumbered(meshgen.tet_cube(9), 3)),
    "elastic1": lambda: elastic_problem(meshgen.hex_cube(1))[::3],
    "elastic8": lambda: elastic_problem(meshgen.hex_cube(8))[::3],
    "tet6_dofs2": lambda: _dofs(meshgen.tet_cube(6), 2),
    "hex5_dofs4": lambda: _dofs(meshgen.hex_cube(5), 4),
}


def _matrix(ctx, monkeypatch, p, v, ranges):
    monkeypatch.setenv("EGPU_TRI_MODE", "range")
    monkeypatch.setenv("EGPU_TRI_RANGES", str(ranges))
    if p.dofs > 1:
        monkeypatch.setenv("EGPU_TRI_NODE_BLOCKS", "1")
    return eg.Matrix(ctx, eg.CRSPattern(p.n, p.nnz, p.dofs, p.perm, p.rows, p.cols, p.diag), v)


@pytest.mark.parametrize("ranges", [3, 148])
@pytest.mark.parametrize("name", list(CASES))
def test_lu_precondition(ctx, monkeypatch, name, ranges):
    p, v = CASES[name]()
    A = _matrix(ctx, monkeypatch, p, v, ranges)
    ilu, _ = A.ilu0(scale_system=True)
    vs = v.copy()
    oracle.scale(p, vs)
    ref = oracle.ilu0(p, vs)
    assert np.array_equal(ilu, ref)
    for seed in (3, 4):
        b = np.random.default_rng(seed).standard_normal(p.n)
        assert rel(A.lu_precondition(b), oracle.lusolve(p, ref, b)) < 1e-13


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("method", [eg.CG, eg.BICGSTAB, eg.GCR, eg.BICGSTABL], ids=["cg", "bicgstab", "gcr", "bicgstabl"])
@pytest.mark.parametrize("name", ["hex10", "hex32", "elastic8"])
def test_solves(ctx, monkeypatch, name, method, precision):
    if method == eg.CG and name == "elastic8":
        pytest.skip("the elasticity system is solved with BiCGStab")
    p, _, _, v, b, _ = elastic_problem(meshgen.hex_cube(8)) if name == "elastic8" else \
        poisson_problem(meshgen.hex_cube(10 if name == "hex10" else 32))
    tol = 1e-12 if precision == "mixed" else 1e-10
    extra = {"restart": 4} if method == eg.BICGSTABL else {}
    x_ref, r_ref = oracle.solve(p, v, b, method=method, precond=eg.PREC_ILU0, max_iter=3000, tol=tol, **extra)
    assert r_ref["info"] == 1
    A = _matrix(ctx, monkeypatch, p, v, 20)
    x, r = A.solve(b, params=eg.SolverParams(method=method, precond=eg.PREC_ILU0, max_iter=3000, tol=tol,
                                             precision=eg.MIXED if precision == "mixed" else eg.FP64, **extra))
    assert r["info"] == 1
    if precision == "fp64":
        assert abs(r["iters"] - r_ref["iters"]) <= 1, (r["iters"], r_ref["iters"])
    assert rel(x, x_ref) < 1e-8


def test_ilu1_rows(ctx, monkeypatch):
    """ILU(1) of the 27-point stencil: up to 62 entries on either side of the diagonal."""
    p, _, _, v, b, _ = poisson_problem(meshgen.hex_cube(8))
    A = _matrix(ctx, monkeypatch, p, v, 20)
    prm = dict(method=eg.BICGSTAB, precond=eg.PREC_ILU0, max_iter=1000, tol=1e-10, ilu_order=1)
    x, r = A.solve(b, params=eg.SolverParams(**prm))
    x_ref, r_ref = oracle.solve(p, v, b, **prm)
    assert r["info"] == 1 and abs(r["iters"] - r_ref["iters"]) <= 1
    assert rel(x, x_ref) < 1e-8
