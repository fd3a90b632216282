"""The L2 projections on the device at the edges of their launch: fewer nodes
than one CTA's rows, node counts that leave a CTA a partial chunk, rules of 4 to
64 points (one to two passes of a warp), and the hull force over 1 to all panels.

Tolerances: both sides solve the mass matrix to a relative residual of 1e-15;
with the condition number of a Q1 mass matrix after Jacobi scaling (below 100 on
these meshes) the fields agree to 1e-12 of the largest entry. The force is a
sum of positive and negative panel values: 1e-13 of the sum of their sizes."""
import numpy as np
import pytest

import oracle as O
from helpers import cube_mesh, relmax
from wavebem_gb300 import meshes as M
from wavebem_gb300.bem_problem import BEMProblem

pytestmark = pytest.mark.gpu


def _mesh(kind, n):
    if kind == "cube":
        X, cells, _ = cube_mesh(n)
        return X, cells, np.ones(len(X), np.uint8)
    m = M.wigley_mesh(n) if kind == "tank" else M.cube_sphere_mesh(n)
    return m.X, m.cells, m.dirichlet


@pytest.mark.parametrize("kind,n", [("cube", 1), ("sphere", 3), ("cube", 4), ("tank", 600), ("tank", 3001), ("tank", 5003)])
@pytest.mark.parametrize("order", [2, 4, 6])
def test_normals_and_gradients_against_the_oracle(kind, n, order):
    X, cells, mask = _mesh(kind, n)
    ptr, idx = M.double_nodes(X, cells)
    P = O.Problem(X, cells, ptr, idx, mask, qorder=order)
    g = BEMProblem(X, cells, mask, ptr, idx, quadrature_order=order)
    g.assemble_system()
    b = np.random.default_rng(n).normal(size=len(X))
    for _ in range(2):  # the buffers are kept
        assert relmax(g.compute_normals(), P.node_normals()) <= 1e-12
        assert relmax(g.compute_surface_gradients(b), P.surface_gradients(b)) <= 1e-12
    assert np.all(g.compute_surface_gradients(np.zeros(len(X))) == 0.0)


def test_hull_force_over_growing_panel_lists():
    X, cells, mask = _mesh("tank", 600)
    ptr, idx = M.double_nodes(X, cells)
    P = O.Problem(X, cells, ptr, idx, mask)
    g = BEMProblem(X, cells, mask, ptr, idx)
    rng = np.random.default_rng(1)
    phi, dn = rng.normal(size=len(X)), rng.normal(size=len(X))
    parts = [abs(P.hull_force(cells[k:k + 1], phi, dn)) for k in range(len(cells))]
    for n in (0, 1, 7, 8, 9, len(cells), 3):
        hull = np.arange(n, dtype=np.int32)
        got = g.hull_force(hull, phi, dn)
        want = P.hull_force(cells[:n], phi, dn) if n else 0.0
        assert abs(got - want) <= 1e-13 * sum(parts[:n])
