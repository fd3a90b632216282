"""The factorisation by the number of 512-column outer panels: two to eight of them,
last panels of a few columns and full ones, last blocks of odd sizes.

Tolerance as for the N = 2,000 factors: TF32 updates keep 11 significant bits
per operand; the entries of L are below 1 and those of U below 1.5 max |S|, so
that S - LU stays below 1e-4 max |S|."""
import numpy as np
import pytest

from wavebem_gb300 import meshes as M
from wavebem_gb300.bem_problem import PREC_MIXED, SOLVER_LU, BEMProblem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [520, 1030, 1100, 1540, 2052, 2570, 3001, 4090])
def test_factor_residual_by_panel_count(n):
    m = M.wigley_mesh(n)
    g = BEMProblem(m.X, m.cells, m.dirichlet, precision=PREC_MIXED, solver=SOLVER_LU)
    g.assemble_system()
    S, LU, perm = g.lu_factors()
    L = np.tril(LU.astype(np.float64), -1) + np.eye(m.n_dofs)
    U = np.triu(LU.astype(np.float64))
    assert np.abs(S - L @ U).max() <= 1e-4 * np.abs(S).max()
    assert np.abs(U).max() <= 1.5 * np.abs(S).max()
    b = M.wigley_bc(m, seed=1)
    phi, dphi = b.copy(), b.copy()
    g.solve(phi, dphi, b)
    assert g.stats()["iterations"] <= 20
