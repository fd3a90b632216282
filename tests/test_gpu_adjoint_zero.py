"""An objective without derivatives: its multipliers are zero, its gradients are
zeros, and the rows without a multiplier are not worked on (the tile kernel is
three quarters of the plain form's adjoint at this size: half the time of a
random objective leaves ample room)."""
import time

import numpy as np
import pytest

from wavebem_gb300 import meshes as M
from wavebem_gb300.bem_problem import PREC_FP64, PREC_MIXED, BEMProblem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED])
def test_zero_objective(precision):
    m = M.wigley_mesh(3001)
    ptr, idx = M.double_nodes(m.X, m.cells)
    b = M.wigley_bc(m, seed=3)
    g = BEMProblem(m.X, m.cells, m.dirichlet, ptr, idx, precision=precision)
    phi, dn = b.copy(), b.copy()
    g.solve(phi, dn, b)

    def timed(J):
        t = []
        for _ in range(5):
            t0 = time.perf_counter()
            out = g.adjoint(J, J)
            t.append(time.perf_counter() - t0)
        return out, sorted(t)[2]

    (gX, gb), zero = timed(np.zeros(m.n_dofs))
    assert not np.any(gX) and not np.any(gb)
    _, full = timed(np.random.default_rng(1).normal(size=m.n_dofs))
    if precision == PREC_FP64:
        assert zero <= 0.5 * full
    g.close()
