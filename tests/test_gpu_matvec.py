"""Mat-vecs of the assembled operators at every remainder of the dof count
modulo the kernels' column steps and rows per CTA (odd counts take the 8-byte
path of the mixed form), against the exported matrices.

Tolerances, relative to sum_j |A_ij x_j| per row: FP64 sums of n terms 1e-15 n;
double-float products and sums 2^-46 a term, bounded by 1e-13."""
import numpy as np
import pytest

from wavebem_gb300 import meshes as M
from wavebem_gb300.bem_problem import PREC_FP64, PREC_MIXED, SOLVER_GMRES_IR, SOLVER_LU, BEMProblem

pytestmark = pytest.mark.gpu

RESOLUTIONS = [(1, 3, 1, 1, 2, 3), (2, 4, 2, 1, 2, 1), (2, 3, 1, 2, 2, 1), (1, 2, 1, 2, 3, 1),
               (10, 10, 19, 15, 3, 11)]  # 136, 137, 134, 123 and 3,001 dofs


@pytest.mark.parametrize("res", RESOLUTIONS)
@pytest.mark.parametrize("prec", [PREC_FP64, PREC_MIXED])
def test_vmult_and_rhs_against_the_matrices(res, prec):
    m = M.wigley_mesh(resolution=res)
    tol = 1e-13 + (1e-15 * m.n_dofs if prec == PREC_FP64 else 0.0)
    g = BEMProblem(m.X, m.cells, m.dirichlet, precision=prec)
    g.assemble_system()
    Nm, Dm = g.matrices()
    a, d = g.compute_alpha(), m.dirichlet.astype(bool)
    v = np.random.default_rng(m.n_dofs).normal(size=m.n_dofs)
    phi, dn = np.where(d, 0.0, v), np.where(d, v, 0.0)
    size = np.abs(Nm) @ np.abs(v) + np.abs(Dm) @ np.abs(v) + np.abs(a * v)
    assert np.all(np.abs(g.vmult(v) - (Nm @ phi + a * phi - Dm @ dn)) <= tol * size)
    phi, dn = np.where(d, v, 0.0), np.where(d, 0.0, v)
    assert np.all(np.abs(g.compute_rhs(v) - (Dm @ dn - Nm @ phi - a * phi)) <= tol * size)


@pytest.mark.parametrize("res", RESOLUTIONS)
def test_refinement_on_the_fp32_system(res):
    """The refinement's inner operator at the same counts: its solution is the
    LU form's (both refine to the same operator, 1e-8 as in every solve)."""
    m = M.wigley_mesh(resolution=res)
    b = M.wigley_bc(m, seed=1)
    got = []
    for solver in (SOLVER_LU, SOLVER_GMRES_IR):
        g = BEMProblem(m.X, m.cells, m.dirichlet, precision=PREC_MIXED, solver=solver)
        phi, dphi = b.copy(), b.copy()
        g.solve(phi, dphi, b)
        got.append(np.concatenate([phi, dphi]))
    assert np.linalg.norm(got[1] - got[0]) <= 1e-8 * np.linalg.norm(got[0])
