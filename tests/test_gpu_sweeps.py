"""The four triangular sweeps at the edges of their block rows: one block, a
last block of a few rows, of odd sizes and full, against FP64 triangular solves
with the same factors.

Tolerance: that of the sweeps with the N = 2,000 factors, 1e-6 of the norm (FP32
substitution, 2^-24 times the growth of factors without pivoting whose system's
diagonal dominates)."""
import numpy as np
import pytest
import scipy.linalg as sl

from helpers import rel2
from wavebem_gb300 import meshes as M
from wavebem_gb300.bem_problem import PREC_MIXED, SOLVER_LU, BEMProblem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [80, 128, 130, 257, 383, 384, 1001, 1300])
def test_sweeps_against_fp64_triangles(n):
    m = M.wigley_mesh(n)
    g = BEMProblem(m.X, m.cells, m.dirichlet, precision=PREC_MIXED, solver=SOLVER_LU)
    g.assemble_system()
    _, LU, _ = g.lu_factors()
    LU = LU.astype(np.float64)
    v = np.random.default_rng(n).normal(size=m.n_dofs)
    y = sl.solve_triangular(LU, sl.solve_triangular(LU, v, lower=True, unit_diagonal=True))
    yt = sl.solve_triangular(LU, sl.solve_triangular(LU, v, trans="T"), lower=True, trans="T",
                             unit_diagonal=True)
    assert rel2(g.lu_apply(v), y) <= 1e-6
    assert rel2(g.lu_apply(v, transpose=True), yt) <= 1e-6
    g.close()
