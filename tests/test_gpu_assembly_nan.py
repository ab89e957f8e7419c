"""A mesh with a NaN coordinate: the assembled matrix and right-hand side are NaN where the reference's are
(ElementMetric skips an integration point only for DetG <= TINY, which NaN is not), so that nothing
downstream takes the elements for missing."""
import numpy as np
import pytest

import elmerfem_b200 as eg
import oracle
from elmerfem_b200 import meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dofs", [1, 3])
@pytest.mark.parametrize("mesh", ["hex", "tet"])
def test_nan_coordinate(ctx, mesh, dofs):
    m = meshgen.hex_cube(3) if mesh == "hex" else meshgen.tet_cube(3)
    m.coords = np.array(m.coords, np.float64)
    m.coords[m.nnodes // 2, 1] = np.nan
    p = oracle.create_pattern(m, dofs=dofs)
    A = eg.Matrix(ctx, eg.CRSPattern(p.n, p.nnz, p.dofs, p.perm, p.rows, p.cols, p.diag))
    A.bind_assembly(m)
    if dofs == 1:
        load = np.ones(m.nnodes)
        vals, rhs = oracle.assemble_poisson(m, p, nodal_k=np.ones(m.nnodes), load=load)
        A.assemble_poisson(nodal_k=np.ones(m.nnodes), load=load)
    else:
        bf = (1.0, 2.0, -3.0)
        vals, rhs = oracle.assemble_elastic(m, p, 1.0, 0.3, bf)
        A.assemble_elastic(1.0, 0.3, bf)
    v, b = A.values(), A.rhs()
    assert np.isnan(rhs).any() and not np.isnan(rhs).all()
    assert np.array_equal(np.isnan(v), np.isnan(vals))
    assert np.array_equal(np.isnan(b), np.isnan(rhs))
    keep = ~np.isnan(rhs)
    assert np.max(np.abs(b[keep] - rhs[keep])) <= 1e-13 * np.max(np.abs(rhs[keep]))
    A.free()
