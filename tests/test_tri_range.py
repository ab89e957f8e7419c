"""The plan of the row-range triangular solves, replayed on the CPU (tests/cpu_model/range_model.cpp):
every value a level reads is an earlier level's, or an external one that its range fetches, whatever
the range size, and the packed entries reproduce CRS_LUSolve (fem/src/CRSMatrix.src:3346-3363)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

import oracle
from elmerfem_b200 import meshgen
from helpers import elastic_problem, poisson_problem, renumbered

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    so = tmp_path_factory.mktemp("range") / "range_model.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-Wall", "-Wextra", "-o", str(so),
                    os.path.join(HERE, "cpu_model", "range_model.cpp")], check=True)
    lib = C.CDLL(str(so))
    i32, f64 = np.ctypeslib.ndpointer(np.int32), np.ctypeslib.ndpointer(np.float64)
    lib.range_replay.argtypes = [C.c_int] * 3 + [i32, i32, i32, f64, f64, f64]
    return lib


def _arrow():
    """A last row with 199 entries: beyond what a row's lanes hold, so the form is not offered."""
    n = 200
    rows = np.concatenate([[1], 1 + np.cumsum([2] * (n - 1) + [n])]).astype(np.int32)
    cols = np.concatenate([[i + 1, n] for i in range(n - 1)] + [np.arange(1, n + 1)]).astype(np.int32)
    p = oracle.create_pattern(meshgen.hex_cube(2))
    p.n, p.rows, p.cols, p.nnz = n, rows, cols, cols.size
    p.diag = np.array([rows[i] if i < n - 1 else rows[n] - 1 for i in range(n)], np.int32)
    v = np.random.default_rng(1).uniform(-1.0, 1.0, cols.size)
    v[p.diag - 1] = 300.0
    return p, v


CASES = {
    "hex6": (lambda: (lambda t: (t[0], t[3]))(poisson_problem(meshgen.hex_cube(6))), 1),
    "hex40": (lambda: (lambda t: (t[0], t[3]))(poisson_problem(meshgen.hex_cube(40, 40, 8))), 1),
    "tet7_renumbered": (lambda: (lambda t: (t[0], t[3]))(poisson_problem(renumbered(meshgen.tet_cube(7), 3))), 1),
    "arrow": (_arrow, 1),
    "elastic4": (lambda: (lambda t: (t[0], t[3]))(elastic_problem(meshgen.hex_cube(4))), 3),
    "hex3_dofs2": (lambda: _dofs(2), 2),
    "hex3_dofs4": (lambda: _dofs(4), 4),
}


def _dofs(dofs):
    p = oracle.create_pattern(meshgen.hex_cube(3), dofs=dofs)
    v = np.random.default_rng(5).uniform(-1.0, 1.0, p.nnz)
    v[p.diag - 1] = np.diff(p.rows).astype(np.float64) + 1.0
    return p, v


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("parts", [1, 3, 148])
def test_replay(model, name, parts):
    make, bs = CASES[name]
    p, v = make()
    vs = v.copy()
    oracle.scale(p, vs)
    ilu = oracle.ilu0(p, vs)
    per = -(-(-(-p.n // parts)) // bs) * bs
    rows, cols, diag = (np.ascontiguousarray(t - 1, np.int32) for t in (p.rows, p.cols, p.diag))
    b = np.random.default_rng(2).standard_normal(p.n)
    z = np.zeros(p.n)
    rc = model.range_replay(p.n, bs, per, rows, cols, diag, ilu, b, z)
    if name == "arrow":
        assert rc == -1
        return
    assert rc == 0
    ref = oracle.lusolve(p, ilu, b)
    # other summation order, and node blocks through their inverses: rounding of short sums
    assert np.linalg.norm(z - ref) <= 1e-13 * np.linalg.norm(ref)
