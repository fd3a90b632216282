"""A vertex of 10,000 panels: set-up and projections take the time of their data,
not of its square (a second here is some hundred times what they need), and the
normals of the flat fan are exact to the solve's 1e-15 residual times the mass
matrix's condition (4 at the diagonal scaling, times the valence's spread:
1e-9)."""
import time

import numpy as np
import pytest

from wavebem_gb300 import meshes as M
from wavebem_gb300.bem_problem import BEMProblem

pytestmark = pytest.mark.gpu


def fan(panels):
    """Quadrilaterals around the origin: centre, two rim points, a point beyond."""
    t = 2 * np.pi * np.arange(2 * panels) / (2 * panels)
    r = np.where(np.arange(2 * panels) % 2, 1.3, 1.0)
    X = np.vstack([[0.0, 0, 0], np.stack([r * np.cos(t), r * np.sin(t), 0 * t], 1)])
    k = 1 + 2 * np.arange(panels)
    nxt = 1 + (2 * np.arange(panels) + 2) % (2 * panels)
    cells = np.stack([0 * k, k, nxt, k + 1], 1).astype(np.int32)
    return X, cells


def test_vertex_of_many_panels():
    warm = M.wigley_mesh(300)
    g = BEMProblem(warm.X, warm.cells, warm.dirichlet)
    g.compute_normals()
    g.close()
    X, cells = fan(10000)
    t0 = time.perf_counter()
    ptr, idx = np.arange(len(X) + 1, dtype=np.int32), np.arange(len(X), dtype=np.int32)
    g = BEMProblem(X, cells, np.ones(len(X), np.uint8), ptr, idx)
    t1 = time.perf_counter()
    n = g.compute_normals()
    t2 = time.perf_counter()
    print("set-up %.3f s, normals %.3f s" % (t1 - t0, t2 - t1))
    assert np.abs(np.asarray(n).reshape(-1, 3) - [0, 0, 1]).max() <= 1e-9
    assert t1 - t0 <= 1.0 and t2 - t1 <= 1.0
    g.close()
