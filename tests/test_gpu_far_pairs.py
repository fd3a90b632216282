"""FP64 assembly where panel and row are far apart: centre terms in 64 bits plus
a remainder in pairs of FP32 numbers, in two forms by distance, and the ways
out of it (panels too small for FP32's exponents, rules of one and two points).

Tolerance: a pair's remainder is at most 2/6 of its entries and is carried to
48 bits through some four roundings in sequence, 2/6 * 4 * 2^-48 = 5e-15 of the
panel's own entries; up to four panels add to an entry, so 1e-14 of D_ij for D.
N's panel terms are as large as D's over the distance where R . n does not
cancel, so 1e-14 of D_ij / |x_i - x_j| for N, doubled for the distance from the
panel instead of the vertex (at least 5/6 of it). The mesh's unit changes D by
its power of two and N not at all: to the last bit. Blocks between a body and one
2^-22 its size, whose panels are below the range of the pairs: 1e-10 of the
block's largest entry, as for the default rules."""
import numpy as np
import pytest

import oracle as O
from helpers import relmax
from wavebem_gb300 import meshes as M
from wavebem_gb300.bem_problem import PREC_FP64, BEMProblem

pytestmark = pytest.mark.gpu

MESHES = {"tank": lambda: M.wigley_mesh(600), "sphere": lambda: M.cube_sphere_mesh(9),
          "cube": lambda: M.cube_sphere_mesh(2)}


def _matrices(m, X, order, oracle=True):
    ptr, idx = M.double_nodes(m.X, m.cells)
    g = BEMProblem(X, m.cells, m.dirichlet, ptr, idx, precision=PREC_FP64, quadrature_order=order)
    g.assemble_system()
    Nm, Dm = g.matrices()
    g.close()
    if not oracle:
        return Nm, Dm
    P = O.Problem(X, m.cells, ptr, idx, m.dirichlet, qorder=order)
    P.assemble()
    return Nm, Dm, P


@pytest.mark.parametrize("mesh", MESHES)
@pytest.mark.parametrize("order", [1, 2, 3, 4, 5, 6])
def test_far_entries(mesh, order):
    m = MESHES[mesh]()
    Nm, Dm, P = _matrices(m, m.X, order)
    r = np.linalg.norm(m.X[:, None] - m.X[None], axis=2)
    h = np.zeros(m.n_dofs)  # largest centre-vertex distance of a vertex's panels
    Pc = m.X[m.cells]
    np.maximum.at(h, m.cells, np.linalg.norm(Pc - Pc.mean(1, keepdims=True), axis=2).max(1)[:, None])
    far = r > 7.0 * h[None]
    assert (mesh == "cube") == (not far.any())
    if far.any():
        assert np.abs((Dm - P.Dm)[far] / P.Dm[far]).max() <= 1e-14
        assert np.abs((Nm - P.Nm)[far] * r[far] / P.Dm[far]).max() <= 2e-14
    assert relmax(Nm, P.Nm) <= 1e-10 and relmax(Dm, P.Dm) <= 1e-10


@pytest.mark.parametrize("power", [-60, -9, 31, 90])
def test_any_unit_of_length(power):
    m = MESHES["tank"]()
    s = 2.0 ** power
    N0, D0 = _matrices(m, m.X, 4, oracle=False)
    N1, D1 = _matrices(m, m.X * s, 4, oracle=False)
    assert np.array_equal(N0, N1) and np.array_equal(D0 * s, D1)


@pytest.mark.parametrize("radius", [2.0 ** -12, 2.0 ** -22])
def test_small_body_in_a_large_one(radius):
    m = M.cube_sphere_mesh(4)
    n = m.n_dofs
    ptr, idx = M.double_nodes(m.X, m.cells)
    X = np.concatenate([m.X, m.X * radius])
    cells = np.concatenate([m.cells, m.cells + n])
    ptr, idx = np.concatenate([ptr, ptr[1:] + ptr[-1]]), np.concatenate([idx, idx + n])
    mask = np.concatenate([m.dirichlet, m.dirichlet])
    g = BEMProblem(X, cells, mask, ptr, idx, precision=PREC_FP64)
    g.assemble_system()
    Nm, Dm = g.matrices()
    g.close()
    P = O.Problem(X, cells, ptr, idx, mask)
    P.assemble()
    for rows in (slice(0, n), slice(n, None)):
        for cols in (slice(0, n), slice(n, None)):
            assert relmax(Nm[rows, cols], P.Nm[rows, cols]) <= 1e-10
            assert relmax(Dm[rows, cols], P.Dm[rows, cols]) <= 1e-10
