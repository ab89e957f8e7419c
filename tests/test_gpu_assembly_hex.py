"""Hexahedral assembly on the FP64 matrix instruction (four elements a warp, groups of elements by
row range and colour) against the oracle: ragged groups, distorted elements, every material
form, and a mesh whose Values span more than one row range."""
import numpy as np
import pytest

import elmerfem_b200 as eg
import oracle
from elmerfem_b200 import meshgen
from helpers import renumbered, row_rel_max

pytestmark = pytest.mark.gpu


def _distorted(mesh, seed):
    rng = np.random.default_rng(seed)
    m = max(mesh.dims) if mesh.dims else round(mesh.nnodes ** (1 / 3)) - 1
    mesh.coords = mesh.coords + rng.uniform(-0.15, 0.15, mesh.coords.shape) / m
    return mesh


MESHES = {
    "one": lambda: meshgen.hex_cube(1),
    "hex2x1x3": lambda: meshgen.hex_cube(2, 1, 3),
    "hex3": lambda: meshgen.hex_cube(3),
    "hex7x5x6": lambda: meshgen.hex_cube(7, 5, 6),
    "hex6_renumbered": lambda: renumbered(meshgen.hex_cube(6), 4),
    "hex75": lambda: meshgen.hex_cube(75),  # 92 MB of Values: two row ranges
}


def _pattern(p):
    return eg.CRSPattern(p.n, p.nnz, p.dofs, p.perm, p.rows, p.cols, p.diag)


@pytest.mark.parametrize("material", ["elem_k", "nodal_k", "unit"])
@pytest.mark.parametrize("name", list(MESHES))
def test_poisson(ctx, name, material):
    m = _distorted(MESHES[name](), 3)
    rng = np.random.default_rng(1)
    ek = np.exp(rng.normal(size=m.nelem)) if material == "elem_k" else None
    nk = np.exp(rng.normal(size=m.nnodes)) if material == "nodal_k" else (np.ones(m.nnodes) if ek is None else None)
    load = rng.uniform(-1.0, 1.0, m.nnodes) if material != "unit" else None
    p = oracle.create_pattern(m)
    vals, rhs = oracle.assemble_poisson(m, p, elem_k=ek, nodal_k=nk, load=np.zeros(m.nnodes) if load is None else load)
    A = eg.Matrix(ctx, _pattern(p))
    A.bind_assembly(m)
    for _ in range(2):  # a second assembly starts from zero again
        A.assemble_poisson(elem_k=ek, nodal_k=None if material == "unit" else nk, load=load)
    assert row_rel_max(p, A.values(), vals) < 1e-13
    assert np.max(np.abs(A.rhs() - rhs)) <= 1e-13 * max(np.max(np.abs(rhs)), 1e-300)


@pytest.mark.parametrize("name", ["one", "hex2x1x3", "hex3", "hex7x5x6", "hex6_renumbered"])
def test_elastic(ctx, name):
    m = _distorted(MESHES[name](), 5)
    p = oracle.create_pattern(m, dofs=3)
    bf = (3.0, -2.0, -1e4)
    vals, rhs = oracle.assemble_elastic(m, p, 200e9, 0.3, bf)
    A = eg.Matrix(ctx, _pattern(p))
    A.bind_assembly(m)
    A.assemble_elastic(200e9, 0.3, bf)
    assert row_rel_max(p, A.values(), vals) < 1e-13
    assert np.max(np.abs(A.rhs() - rhs)) <= 1e-13 * np.max(np.abs(rhs))


@pytest.mark.parametrize("symmetric", [False, True])
def test_dirichlet_values(ctx, symmetric):
    """Rows of every length against the oracle, with non-zero boundary values."""
    m = _distorted(meshgen.hex_cube(7, 5, 6), 2)
    p = oracle.create_pattern(m)
    vals, rhs = oracle.assemble_poisson(m, p, nodal_k=np.ones(m.nnodes), load=np.ones(m.nnodes))
    con = np.sort(p.perm[m.boundary_nodes([1, 4, 5]) - 1]).astype(np.int32)
    cv = np.random.default_rng(3).uniform(-2.0, 2.0, con.size)
    v, b = vals.copy(), rhs.copy()
    oracle.dirichlet(p, v, b, con, cv, symmetric=symmetric)
    A = eg.Matrix(ctx, _pattern(p))
    A.bind_assembly(m)
    A.assemble_poisson(load=np.ones(m.nnodes))
    A.dirichlet(con, cv, symmetric=symmetric)
    assert row_rel_max(p, A.values(), v) < 1e-13
    assert np.max(np.abs(A.rhs() - b)) <= 1e-12 * np.max(np.abs(b))
