"""Rows of every width class in the kernels that unroll over them: the product (lane groups of 4 to
32, two rows each, four entries a lane before the remainder loop), the SELL loops of the Krylov
solves (whole rows of 9, chunks of 5, shared offset lists in chunks of 32, absolute columns), the
FP64 residual of the mixed solve and the batched solver, at grids of one block and of several.

Product: each row is a sum of len products in some order, so it is within (len + 2) eps of
sum |a||x| (the textbook bound of a dot product).  Solves: the matrices are diagonally dominant,
a_ii >= 1 + sum_j |a_ij|, so the scaled matrix S = D A D has eigenvalues in [1/max a_ii, 2], and a
scaled residual ||D (b - A x)|| <= tol ||D b|| bounds the error of x; the check is on that residual,
taken here in FP64, with 2x for the recursive residual's own rounding.
"""
import numpy as np
import pytest

import elmerfem_b200 as eg

pytestmark = pytest.mark.gpu


def _matrix(n, lists, symmetric_band=None, seed=0):
    """CRS pattern (1-based, sorted, with the diagonal) and dominant values from column lists."""
    rng = np.random.default_rng(seed)
    rows, cols, vals, diag = [1], [], [], []
    for i, js in enumerate(lists):
        js = sorted(set(js) | {i})
        a = np.array([_pair(seed, min(i, j), max(i, j)) if symmetric_band else rng.uniform(-1, 1) for j in js])
        d = js.index(i)
        a[d] = 1.5 + np.abs(a).sum() - abs(a[d])
        diag.append(len(cols) + d + 1)
        cols += [j + 1 for j in js]
        vals += list(a)
        rows.append(len(cols) + 1)
    i32 = lambda q: np.array(q, np.int32)
    p = eg.CRSPattern(n, len(cols), 1, np.arange(1, n + 1, dtype=np.int32), i32(rows), i32(cols), i32(diag))
    return p, np.array(vals)


def _pair(seed, i, j):
    return np.sin(1.0 + 12.9898 * i + 78.233 * j + seed)


def _dot(p, v, x):
    s = np.zeros(p.n)
    np.add.at(s, np.repeat(np.arange(p.n), np.diff(p.rows)), v * x[p.cols - 1])
    return s


@pytest.mark.parametrize("n", [1, 2, 3, 33, 257])
@pytest.mark.parametrize("width", [1, 5, 17, 40, 130])
def test_product(ctx, n, width):
    rng = np.random.default_rng(n * 1000 + width)
    lists = [list(rng.choice(n, size=min(n, 1 + (i * 7) % width), replace=False)) for i in range(n)]
    p, v = _matrix(n, lists, seed=width)
    x = rng.standard_normal(n)
    y = eg.Matrix(ctx, p, v).mv(x)
    scale = _dot(p, np.abs(v), np.abs(x))
    lens = np.diff(p.rows)
    assert np.all(np.abs(y - _dot(p, v, x)) <= 2 * (lens + 2) * np.finfo(float).eps * scale)


def _band(n, half):
    return [list(range(max(0, i - half), min(n, i + half + 1))) for i in range(n)]


def _scattered(n, half):
    lists = [set() for _ in range(n)]
    rng = np.random.default_rng(half)
    for i in range(n):
        for j in rng.choice(n, size=min(n, half), replace=False):
            lists[i].add(int(j))
            lists[int(j)].add(i)
    return [sorted(s) for s in lists]


def _far(n, half):
    """tridiagonal plus couplings beyond 16-bit offsets"""
    return [[j for j in (i - 1, i + 1, i - 33000, i + 33000) if 0 <= j < n] for i in range(n)]


# half widths: rows of 3, 9, 13, 27, 45 and 71 entries where the band is whole; n: one block of 16
# slices, one more, and 4 blocks with a partial slice
@pytest.mark.parametrize("make,n,half", [(_band, 512, h) for h in (1, 4, 6, 13, 22, 35)]
                         + [(_band, 513, 4), (_band, 1601, 13), (_band, 1601, 6), (_scattered, 512, 2),
                            (_scattered, 1601, 6), (_scattered, 1601, 14), (_far, 40001, 1)])
@pytest.mark.parametrize("method", [eg.CG, eg.BICGSTAB], ids=["cg", "bicgstab"])
def test_solves(ctx, make, n, half, method):
    p, v = _matrix(n, make(n, half), symmetric_band=True, seed=half)
    b = np.random.default_rng(n).uniform(-1, 1, n)
    tol = 1e-10
    D = 1.0 / np.sqrt(v[p.diag - 1])
    bound = 2 * tol * np.linalg.norm(D * b)
    A = eg.Matrix(ctx, p, v)
    for precision in (eg.FP64, eg.MIXED):
        x, r = A.solve(b, params=eg.SolverParams(method=method, precond=eg.PREC_DIAGONAL, max_iter=500, tol=tol,
                                                 precision=precision))
        assert r["info"] == 1
        assert np.linalg.norm(D * (b - _dot(p, v, x))) <= bound
    # the batch takes ILU0 (here by two Jacobi sweeps a triangle) with BiCGStab only
    for prec in (eg.PREC_DIAGONAL, eg.PREC_ILU0)[:1 if method == eg.CG else 2]:
        B = eg.Batch(ctx, eg.SolverParams(method=method, precond=prec, max_iter=500, tol=tol, ilu_sweeps=2))
        try:
            i = B.add(p, v, b)
            B.solve()
            assert B.result(i)["info"] == 1
            x = B.solution(i)
        finally:
            B.free()
        assert np.linalg.norm(D * (b - _dot(p, v, x))) <= bound
