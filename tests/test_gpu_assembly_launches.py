"""One launch per element colour, whatever the size and the numbering of the mesh (cutting a colour into
ranges of rows made every assembly slower)."""
import numpy as np
import pytest

import elmerfem_b200 as eg
from elmerfem_b200 import meshgen

pytestmark = pytest.mark.gpu


def _launches(ctx, mesh, dofs):
    A = eg.Matrix(ctx, eg.create_matrix(mesh, dofs=dofs))
    A.bind_assembly(mesh)
    n0 = ctx.kernel_launches
    if dofs == 1:
        A.assemble_poisson(load=np.ones(mesh.nnodes))
    else:
        A.assemble_elastic(1.0, 0.3, (0.0, 0.0, 1.0))
    n = ctx.kernel_launches - n0
    A.free()
    return n


@pytest.mark.parametrize("cube,dofs,cells", [(meshgen.hex_cube, 1, 75), (meshgen.hex_cube, 3, 36)],
                         ids=["poisson", "elastic"])
def test_launches_do_not_grow_with_the_mesh(ctx, cube, dofs, cells):
    """92 MB and 93 MB of Values: two fills and eight colours, as on a small mesh."""
    assert _launches(ctx, cube(cells), dofs) == _launches(ctx, cube(6), dofs) == 10
