"""Panel records, near, singular and merge kernels at the edges of their lane
layouts: rules of at most 16 points (two panels per warp) and of 25 and 36
(one, in several passes), vertex-singular rules of 18 to 128 points, and a
tank with a panel taken out: its odd panel count leaves half a warp without
one.

Tolerances: FP64 entries 1e-10 of the largest, as for the default rules. Mixed
entries 2e-8: a far entry's FP32 point differences carry a few 2^-24 of the
O(panel / distance <= 1/4) difference terms, at most 1.5e-8 of the largest
entry even where a far entry is as large as a near one."""
import numpy as np
import pytest

import oracle as O
from helpers import relmax
from wavebem_gb300 import meshes as M
from wavebem_gb300.bem_problem import PREC_FP64, PREC_MIXED, BEMProblem

pytestmark = pytest.mark.gpu

MESHES = {"tank": lambda: M.wigley_mesh(resolution=(2, 3, 4, 3, 2, 3)),
          "sphere": lambda: M.cube_sphere_mesh(5)}


@pytest.mark.parametrize("mesh", MESHES)
@pytest.mark.parametrize("order,singular", [(2, 3), (3, 5), (4, 5), (5, 8), (6, 4)])
def test_entries_and_alpha_for_every_rule(mesh, order, singular):
    m = MESHES[mesh]()
    cells = m.cells[:-1] if mesh == "tank" else m.cells
    ptr, idx = M.double_nodes(m.X, cells)
    P = O.Problem(m.X, cells, ptr, idx, m.dirichlet, qorder=order, sorder=singular)
    P.assemble()
    for prec, tol in ((PREC_FP64, 1e-10), (PREC_MIXED, 2e-8)):
        g = BEMProblem(m.X, cells, m.dirichlet, ptr, idx, precision=prec, quadrature_order=order,
                       singular_quadrature_order=singular)
        g.assemble_system()
        Nm, Dm = g.matrices()
        assert relmax(Nm, P.Nm) <= tol and relmax(Dm, P.Dm) <= tol
        assert relmax(g.compute_alpha(), P.alpha) <= tol * m.n_dofs ** 0.5
        g.close()
