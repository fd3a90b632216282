"""The FMA product for every expansion order (27 to 512 nodes: one to four
shares of the M2L's target nodes, the last ones partly empty) and for rules of
4 to 36 points (segments of the near field from a fraction of a chunk on,
blocks of a few rows), against the dense FP64 operators of the same rule.

Tolerance: the default order's measured 1.4e-5, sevenfold per order, times ten
for the coarser tree of this mesh."""
import numpy as np
import pytest

from helpers import rel2
from wavebem_gb300 import meshes as M
from wavebem_gb300.bem_problem import METHOD_FMA, PREC_FP64, BEMProblem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,rule", [(3, 4), (4, 2), (5, 3), (6, 5), (6, 6), (7, 4), (8, 4)])
def test_product_for_every_order_and_rule(order, rule):
    m = M.wigley_mesh(3001)
    ptr, idx = M.double_nodes(m.X, m.cells)
    v = np.random.default_rng(order).normal(size=m.n_dofs)
    g = BEMProblem(m.X, m.cells, m.dirichlet, ptr, idx, precision=PREC_FP64, quadrature_order=rule)
    f = BEMProblem(m.X, m.cells, m.dirichlet, ptr, idx, method=METHOD_FMA, fma_order=order,
                   quadrature_order=rule)
    g.assemble_system()
    f.assemble_system()
    tol = 1.4e-4 * 7.0 ** (6 - order)
    assert rel2(f.vmult(v), g.vmult(v)) <= tol and rel2(f.compute_rhs(v), g.compute_rhs(v)) <= tol
    f.close()
    g.close()
