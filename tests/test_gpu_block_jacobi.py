"""The block-Jacobi preconditioned FP64 solve with last blocks of a few rows, of
odd sizes and full (the apply takes a block in four row groups and four column
quarters), against the CPU oracle's solve.

Tolerance: both solve to a relative residual of 1e-10 or below, and the systems'
condition (a few hundred at these sizes) carries that into the solution: 1e-7."""
import numpy as np
import pytest

import oracle as O
from helpers import rel2
from wavebem_gb300 import meshes as M
from wavebem_gb300.bem_problem import PREC_FP64, BEMProblem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [80, 128, 257, 383, 384])
def test_fp64_solve_by_block_shape(n):
    m = M.wigley_mesh(n)
    ptr, idx = M.double_nodes(m.X, m.cells)
    b = M.wigley_bc(m, seed=n)
    g = BEMProblem(m.X, m.cells, m.dirichlet, ptr, idx, precision=PREC_FP64, tolerance=1e-13)
    g.assemble_system()
    phi, dphi = b.copy(), b.copy()
    g.solve_system(phi, dphi, b)
    P = O.Problem(m.X, m.cells, ptr, idx, m.dirichlet)
    P.assemble()
    pr, dr, _ = P.solve_system(b)
    assert rel2(phi, pr) <= 1e-7 and rel2(dphi, dr) <= 1e-7
    g.close()
