"""A device error word that is set when a solve fails for another reason is what
the call reports, and it is cleared: the next call on the handle starts clean.
The word is preset by a test entry point; no wait is made to run out."""
import numpy as np
import pytest

from wavebem_gb300 import meshes as M
from wavebem_gb300.bem_problem import (PREC_MIXED, SOLVER_GMRES, SOLVER_GMRES_IR, SOLVER_LU, BEMProblem,
                                       NoConvergence, WBEMError)

pytestmark = pytest.mark.gpu
TIMEOUT = 8


@pytest.mark.parametrize("solver", [SOLVER_LU, SOLVER_GMRES, SOLVER_GMRES_IR])
def test_failed_solve_reports_the_word(solver):
    m = M.wigley_mesh(300)
    b = M.wigley_bc(m, seed=2)
    # one step is not enough: every solve ends without convergence
    g = BEMProblem(m.X, m.cells, m.dirichlet, precision=PREC_MIXED, solver=solver, max_steps=1)
    g.assemble_system()
    with pytest.raises(NoConvergence):
        g.solve_system(b.copy(), b.copy(), b)
    assert g.L.wbem_test_device_error(g.h, TIMEOUT) == 0
    with pytest.raises(WBEMError) as e:
        g.solve_system(b.copy(), b.copy(), b)
    assert e.value.code == TIMEOUT
    with pytest.raises(NoConvergence):
        g.solve_system(b.copy(), b.copy(), b)
    assert np.isfinite(g.compute_normals()).all()
    g.close()


@pytest.mark.parametrize("n", [300, 3300])
def test_solve_that_converges_reports_the_word(n):
    """Both forms of the Arnoldi step (one cluster, grid barriers)."""
    m = M.wigley_mesh(n)
    b = M.wigley_bc(m, seed=2)
    g = BEMProblem(m.X, m.cells, m.dirichlet, precision=PREC_MIXED, solver=SOLVER_LU)
    g.assemble_system()
    phi, dn = b.copy(), b.copy()
    g.solve_system(phi, dn, b)
    assert g.L.wbem_test_device_error(g.h, TIMEOUT) == 0
    with pytest.raises(WBEMError) as e:
        g.solve_system(b.copy(), b.copy(), b)
    assert e.value.code == TIMEOUT
    p2, d2 = b.copy(), b.copy()
    g.solve_system(p2, d2, b)
    assert np.array_equal(phi, p2) and np.array_equal(dn, d2)
    g.close()
