"""The multipole method with other rules than the default: a tree that is kept
takes a changed singular rule (equality with a handle that never had another),
and the projections of a handle with 49 and 64 points per panel, which only this
method accepts, against the oracle (1e-12, as for the rules of up to 36)."""
import numpy as np
import pytest

import oracle as O
from helpers import relmax
from wavebem_gb300 import meshes as M
from wavebem_gb300.bem_problem import METHOD_FMA, PREC_MIXED, BEMProblem

pytestmark = pytest.mark.gpu


def handle(m, ptr, idx, order, singular):
    return BEMProblem(m.X, m.cells, m.dirichlet, ptr, idx, precision=PREC_MIXED, method=METHOD_FMA,
                      quadrature_order=order, singular_quadrature_order=singular)


def test_kept_tree_takes_the_singular_rule():
    m = M.wigley_mesh(2000)
    ptr, idx = M.double_nodes(m.X, m.cells)
    v = np.random.default_rng(0).normal(size=m.n_dofs)
    g = handle(m, ptr, idx, 4, 3)
    g.assemble_system()
    first = g.vmult(v).copy()
    g.options.singular_quadrature_order = 7
    g.assemble_system()
    fresh = handle(m, ptr, idx, 4, 7)
    fresh.assemble_system()
    assert np.array_equal(g.vmult(v), fresh.vmult(v))
    assert not np.array_equal(g.vmult(v), first)
    g.close()
    fresh.close()


@pytest.mark.parametrize("order", [7, 8])
def test_projections_of_large_rules(order):
    m = M.wigley_mesh(2000)
    ptr, idx = M.double_nodes(m.X, m.cells)
    P = O.Problem(m.X, m.cells, ptr, idx, m.dirichlet, qorder=order)
    g = handle(m, ptr, idx, order, 5)
    g.assemble_system()
    b = np.random.default_rng(order).normal(size=m.n_dofs)
    assert relmax(g.compute_normals(), P.node_normals()) <= 1e-12
    assert relmax(g.compute_surface_gradients(b), P.surface_gradients(b)) <= 1e-12
    g.close()
