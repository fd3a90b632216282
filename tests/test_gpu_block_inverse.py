"""The inverses of the block-Jacobi blocks, through the number of GMRES steps:
with one block the preconditioner is the inverse of the system, so that one step
solves it; a second block of r rows couples through a matrix of rank 2 r at most,
so that 2 r + 1 steps do. One block of less than 128 rows, of exactly 128, last
blocks of one and two rows; pivots that tie in magnitude (the sphere's
symmetry), pivots off the diagonal (constraint rows of the tank), and rows that
dominate their diagonal (every CTA of the cluster runs out of rows in turn).

Tolerance: n^1.5 eps cond |rhs| <= 128^1.5 1.1e-16 1e3 = 1.6e-10 is left by one
step with an inverse from Gauss-Jordan with partial pivoting; the solve is asked
for 1e-8 and the solution (cond 1e3 at most) compared to 1e-5."""
import numpy as np
import pytest

from helpers import rel2
from wavebem_gb300 import meshes as M
from wavebem_gb300.bem_problem import PREC_FP64, PREC_MIXED, SOLVER_GMRES, BEMProblem

pytestmark = pytest.mark.gpu


def patch(nx, ny):
    """A curved patch of nx x ny nodes, all Dirichlet."""
    u, v = np.meshgrid(np.linspace(0, 1, nx), np.linspace(0, 1, ny))
    u, v = u.ravel(), v.ravel()
    X = np.stack([u, v + 0.1 * u * u, 0.3 * np.sin(2 * u + v)], 1)
    i = (np.arange(nx - 1)[None] + nx * np.arange(ny - 1)[:, None]).ravel()
    cells = np.stack([i, i + 1, i + nx, i + nx + 1], 1).astype(np.int32)
    return X, cells, np.ones(nx * ny, np.uint8)


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED])
@pytest.mark.parametrize("mesh", ["sphere", "tank", (14, 7), (16, 8), (43, 3), (26, 5)])
def test_steps_by_block_shape(mesh, precision):
    if mesh == "sphere":
        m = M.cube_sphere_mesh(4)
        X, cells, mask = m.X, m.cells, m.dirichlet
    elif mesh == "tank":
        m = M.wigley_mesh(100)
        X, cells, mask = m.X, m.cells, m.dirichlet
    else:
        X, cells, mask = patch(*mesh)
    N = len(X)
    assert N == {"sphere": 98, "tank": 100}.get(mesh) or N == mesh[0] * mesh[1]
    g = BEMProblem(X, cells, mask, precision=precision, solver=SOLVER_GMRES, tolerance=1e-8)
    g.assemble_system()
    b = np.random.default_rng(2).normal(size=N)
    phi, dphi = b.copy(), b.copy()
    g.solve_system(phi, dphi, b)
    assert g.stats()["iterations"] <= (1 if N <= 128 else 2 * (N - 128) + 1)
    tight = BEMProblem(X, cells, mask, precision=precision, solver=SOLVER_GMRES, tolerance=1e-13)
    tight.assemble_system()
    pt, dt = b.copy(), b.copy()
    tight.solve_system(pt, dt, b)
    assert rel2(np.r_[phi, dphi], np.r_[pt, dt]) <= 1e-5
    g.close()
    tight.close()
