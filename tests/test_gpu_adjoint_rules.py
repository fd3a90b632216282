"""Adjoint panel terms for every rule: the FP64 form's moments over several
rows per thread (1,001 dofs: two CTAs of rows, the second with half its warps
empty) and the mixed form's near pairs, whose points lie over the lanes of a
half warp (4 and 9 of 16 lanes, two and three points per lane), with
vertex-singular rules of 18 to 128 points.

Tolerances: those of the default rules, FP64 against central differences
(h = 1e-6) 1e-6, mixed against FP64 1e-6."""
import numpy as np
import pytest

from helpers import rel2
from wavebem_gb300 import meshes as M
from wavebem_gb300.bem_problem import PREC_FP64, PREC_MIXED, BEMProblem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,singular", [(2, 3), (3, 5), (5, 8), (6, 4)])
def test_gradient_for_every_rule(order, singular):
    m = M.wigley_mesh(1001)
    ptr, idx = M.double_nodes(m.X, m.cells)
    b = M.wigley_bc(m, seed=3)
    rng = np.random.default_rng(order)
    c, dd = rng.normal(size=m.n_dofs), rng.normal(size=m.n_dofs)

    def solved(X, prec):
        g = BEMProblem(X, m.cells, m.dirichlet, ptr, idx, precision=prec, tolerance=1e-14,
                       quadrature_order=order, singular_quadrature_order=singular)
        phi, dphi = b.copy(), b.copy()
        g.solve(phi, dphi, b)
        return g, float(c @ phi + dd @ dphi)

    g, _ = solved(m.X, PREC_FP64)
    gX, gb = g.adjoint(c, dd)
    A = rng.normal(size=(3, 3))
    d = 0.1 * np.sin(m.X @ A + rng.uniform(0, 2 * np.pi, 3))
    h = 1e-6
    fd = (solved(m.X + h * d, PREC_FP64)[1] - solved(m.X - h * d, PREC_FP64)[1]) / (2 * h)
    assert abs(float(np.sum(gX * d)) - fd) <= 1e-6 * abs(fd)
    gm, _ = solved(m.X, PREC_MIXED)
    gXm, gbm = gm.adjoint(c, dd)
    assert rel2(gXm, gX) <= 1e-6 and rel2(gbm, gb) <= 1e-6
