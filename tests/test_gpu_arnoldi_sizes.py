"""Arnoldi steps on either side of the row count up to which one cluster takes
them (3,200), and with clusters whose last CTAs have few rows or none, against
the CPU oracle's solve.

Tolerance: both solve to a relative residual of 1e-10 or below, and the systems'
condition (a few hundred at these sizes) carries that into the solution: 1e-7."""
import numpy as np
import pytest

import oracle as O
from helpers import rel2
from wavebem_gb300 import meshes as M
from wavebem_gb300.bem_problem import PREC_FP64, BEMProblem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh", ["sphere2", "sphere3", "tank1045", "tank3180", "tank3240"])
def test_solve_by_row_count(mesh):
    if mesh.startswith("sphere"):
        m = M.cube_sphere_mesh(int(mesh[6:]))  # 26 and 56 dofs: two and four rows per CTA
        mask = np.ones(m.n_dofs, np.uint8)
        b = np.random.default_rng(1).normal(size=m.n_dofs)
    else:
        m = M.wigley_mesh(int(mesh[4:]))
        mask, b = m.dirichlet, M.wigley_bc(m, seed=1)
    ptr, idx = M.double_nodes(m.X, m.cells)
    g = BEMProblem(m.X, m.cells, mask, ptr, idx, precision=PREC_FP64, tolerance=1e-13)
    g.assemble_system()
    phi, dphi = b.copy(), b.copy()
    g.solve_system(phi, dphi, b)
    P = O.Problem(m.X, m.cells, ptr, idx, mask)
    P.assemble()
    pr, dr, _ = P.solve_system(b)
    assert rel2(phi, pr) <= 1e-7 and rel2(dphi, dr) <= 1e-7
    g.close()
