"""Two live handles with other quadrature rules: what one returns does not depend
on what the other has been set up with, in one thread or in two. Equality: the
same kernels on the same data."""
import threading

import numpy as np
import pytest

from wavebem_gb300 import meshes as M
from wavebem_gb300.bem_problem import PREC_FP64, PREC_MIXED, BEMProblem

pytestmark = pytest.mark.gpu


def problem(m, order, singular, precision):
    ptr, idx = M.double_nodes(m.X, m.cells)
    return BEMProblem(m.X, m.cells, m.dirichlet, ptr, idx, precision=precision, quadrature_order=order,
                      singular_quadrature_order=singular)


def results(g, m, hull, b):
    phi, dn = b.copy(), b.copy()
    g.solve(phi, dn, b)
    gX, gb = g.force_adjoint(hull, b)
    return [phi, dn, gX, gb, np.array(g.hull_force(hull, phi, dn)), g.compute_normals()]


@pytest.mark.parametrize("precision", [PREC_MIXED, PREC_FP64])
@pytest.mark.parametrize("order,singular", [(6, 5), (3, 7)])
def test_another_handle_with_another_rule(precision, order, singular):
    m = M.wigley_mesh(300)
    hull = np.nonzero(m.face == M.HULL)[0].astype(np.int32)
    b = M.wigley_bc(m, seed=4)
    a = problem(m, order, singular, precision)
    first = results(a, m, hull, b)
    other = problem(m, 4, 5, precision)  # creating it sets its rule up
    phi, dn = first[0], first[1]
    gX, gb = a.force_adjoint(hull, b)
    assert np.array_equal(gX, first[2]) and np.array_equal(gb, first[3])
    assert a.hull_force(hull, phi, dn) == float(first[4])
    other.solve(b.copy(), b.copy(), b)
    assert a.hull_force(hull, phi, dn) == float(first[4])
    a.close()
    other.close()


def test_two_threads_with_other_rules():
    m = M.wigley_mesh(600)
    hull = np.nonzero(m.face == M.HULL)[0].astype(np.int32)
    b = M.wigley_bc(m, seed=5)
    rules = [(6, 5), (3, 7)]
    alone = []
    for o, s in rules:
        g = problem(m, o, s, PREC_MIXED)
        alone.append(results(g, m, hull, b))
        g.close()
    wrong = []

    def work(k):
        g = problem(m, *rules[k], PREC_MIXED)
        for n in range(10):
            for x, y in zip(results(g, m, hull, b), alone[k]):
                if not np.array_equal(x, y):
                    wrong.append((k, n))
        g.close()

    ts = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not wrong
