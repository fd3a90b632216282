"""The mixed operators on both sides of the size up to which a CTA splits the
vector itself (1,500 columns), even and odd, against the decoded matrices in
FP64. Tolerance: products of pairs of floats, 48 bits each, summed in such pairs
over at most six terms and in FP64 beyond: 1e-13 of the sum of magnitudes."""
import numpy as np
import pytest

from wavebem_gb300.bem_problem import PREC_MIXED, BEMProblem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(2, 2), (7, 43), (14, 107), (50, 30), (79, 19), (38, 40)])
def test_products_around_the_line(nx, ny):
    u, v = np.meshgrid(np.linspace(0, 1, nx), np.linspace(0, 1, ny))
    u, v = u.ravel(), v.ravel()
    X = np.stack([u, v + 0.1 * u * u, 0.3 * np.sin(2 * u + v)], 1)
    i = (np.arange(nx - 1)[None] + nx * np.arange(ny - 1)[:, None]).ravel()
    cells = np.stack([i, i + 1, i + nx, i + nx + 1], 1).astype(np.int32)
    N = nx * ny
    rng = np.random.default_rng(N)
    mask = (rng.random(N) < 0.5).astype(np.uint8)
    mask[0] = 1
    ptr, idx = np.arange(N + 1, dtype=np.int32), np.arange(N, dtype=np.int32)
    g = BEMProblem(X, cells, mask, ptr, idx, precision=PREC_MIXED)
    g.assemble_system()
    Nm, Dm = g.matrices()
    a, m, x = g.compute_alpha(), mask.astype(bool), rng.normal(size=N)
    A, B = np.where(m, -Dm, Nm), np.where(m, -Nm, Dm)
    for got, M, diag in ((g.vmult(x), A, np.where(m, 0, a)), (g.compute_rhs(x), B, np.where(m, -a, 0))):
        assert np.all(np.abs(got - (M @ x + diag * x)) <= 1e-13 * (np.abs(M) @ np.abs(x) + np.abs(diag * x)) + 1e-300)
    g.close()
