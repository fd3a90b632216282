"""The order of operations of the FP32 factorisation and of its triangular
sweeps, against an elimination in FP32 on the host, bit for bit: every entry
takes its multiply-subtracts one pivot after the other, ascending; the products
with the blocks' inverses are chains in ascending k; a sweep subtracts block
after block. A refinement that stops at its tolerance after two steps carries
the rounding of the factors into its answer, so the order is part of the result.

Up to 512 columns, where no tensor-core update is involved. The GPU's
approximate reciprocals of the pivots are taken from its own factors: the
candidates within two units in the last place of 1 / pivot, of which one has to
give every multiplier of the column. Equality, no tolerance: each operation is
correctly rounded on both sides."""
import numpy as np
import pytest

from wavebem_gb300 import meshes as M
from wavebem_gb300.bem_problem import PREC_MIXED, SOLVER_LU, BEMProblem

pytestmark = pytest.mark.gpu
f4, B = np.float32, 128


def fma(a, b, c):
    """a b + c of FP32 values, rounded once (the 64-bit sum rounded to odd)."""
    p, c = np.multiply(a, b, dtype=np.float64), np.asarray(c, np.float64)
    s = p + c
    bb = s - p
    e = (p - (s - bb)) + (c - bb)
    odd = (s.view(np.int64) & 1).astype(bool)
    s = np.where((e != 0) & ~odd, np.nextafter(s, np.where(e > 0, np.inf, -np.inf)), s)
    return s.astype(f4)


def chain(P, Q):
    """P Q, each entry one chain of multiply-adds in ascending k."""
    s = np.zeros((P.shape[0], Q.shape[1]), f4)
    for k in range(P.shape[1]):
        s = fma(P[:, k:k + 1], Q[k:k + 1], s)
    return s


def eliminate(S, known):
    """L, U and inv(L) of one block, and for each pivot the reciprocals that
    give known's multipliers."""
    n = len(S)
    W, L, cands = np.hstack([S, np.eye(n, dtype=f4)]), np.eye(n, dtype=f4), []
    for k in range(n):
        r = f4(1.0) / W[k, k]
        near = [r]
        for _ in range(2):
            near = [np.nextafter(near[0], f4(-np.inf))] + near + [np.nextafter(near[-1], f4(np.inf))]
        cands.append([c for c in near if np.array_equal(W[k + 1:, k] * c, known[k + 1:, k])])
        assert cands[-1], f"no reciprocal gives the multipliers of pivot {k}"
        L[k + 1:, k] = W[k + 1:, k] * cands[-1][0]
        W[k + 1:] = fma(-L[k + 1:, k:k + 1], W[k:k + 1], W[k + 1:])
    return L, np.triu(W[:, :n]), np.tril(W[:, n:]), cands


def inv_u_row(U, r, dinv):
    x = np.zeros(len(U), f4)
    x[r] = 1.0
    for k in range(r, len(U)):
        x[k] *= dinv[k]
        x[k + 1:] = fma(-x[k], U[k, k + 1:], x[k + 1:])
    return x


def inv_u(U, cands, A=None, X=None):
    """inv(U) with the reciprocals that give the column panel X = A inv(U)."""
    n = len(U)
    dinv, V, Z = np.zeros(n, f4), np.zeros((n, n), f4), np.eye(n, dtype=f4)
    for k in range(n):
        for c in cands[k]:
            col = Z[:k + 1, k] * c
            if A is None or np.array_equal(chain(A[:, :k + 1], col[:, None])[:, 0], X[:, k]):
                break
        else:
            raise AssertionError(f"no reciprocal gives column {k} of the panel")
        dinv[k], V[:k + 1, k] = c, col
        Z[:k + 1, k + 1:] = fma(-col[:, None], U[k, k + 1:][None], Z[:k + 1, k + 1:])
    return V, dinv


def tree(p):
    """Sum over 32 lanes, halves added pairwise."""
    for o in (16, 8, 4, 2, 1):
        p = p + p[..., np.arange(p.shape[-1]) ^ o]
    return p[..., 0]


def block_dot(T, v, columns):
    """T v of a 128 x 128 block as the sweeps form it."""
    if columns:  # rows over lanes of four columns
        t, x = T.reshape(-1, 32, 4), v.reshape(32, 4)
        s = t[..., 0] * x[:, 0]
        for u in range(1, 4):
            s = fma(t[..., u], x[:, u], s)
        return tree(s)
    out = []  # T given transposed: entries of one parity, four chains each
    for h in range(2):
        q = [np.zeros(len(T), f4) for _ in range(4)]
        for i in range(64):
            q[i % 4] = fma(T[:, h + 2 * i], v[h + 2 * i], q[i % 4])
        out.append((q[0] + q[1]) + (q[2] + q[3]))
    return out[0] + out[1]


def diag_dot(V, a):
    q = [np.zeros(len(V), f4) for _ in range(4)]
    for c in range(len(a)):
        q[c % 4] = fma(V[:, c], a[c], q[c % 4])
    return (q[0] + q[1]) + (q[2] + q[3])


def sweep(T, inv, v, order, columns):
    nb, x = len(inv), {}
    for n, k in enumerate(order):
        a = v[k * B:(k + 1) * B].copy()
        for j in order[:n]:
            a -= block_dot(T[k * B:(k + 1) * B, j * B:(j + 1) * B], x[j], columns)
        x[k] = diag_dot(inv[k], a)
    return np.concatenate([x[k] for k in range(nb)])


def patch(nx, ny):
    """A curved patch of nx x ny nodes."""
    u, v = np.meshgrid(np.linspace(0, 1, nx), np.linspace(0, 1, ny))
    u, v = u.ravel(), v.ravel()
    X = np.stack([u, v + 0.1 * u * u, 0.3 * np.sin(2 * u + v)], 1)
    i = (np.arange(nx - 1)[None] + nx * np.arange(ny - 1)[:, None]).ravel()
    cells = np.stack([i, i + 1, i + nx, i + nx + 1], 1).astype(np.int32)
    return X, cells, np.ones(nx * ny, np.uint8)


# one block of 98, exactly one, one row more, three with a ragged last one, exactly two, a tank
@pytest.mark.parametrize("mesh", [(14, 7), (16, 8), (43, 3), (20, 15), (32, 8), "tank"])
def test_factors_and_sweeps_bitwise(mesh):
    if mesh == "tank":
        m = M.wigley_mesh(400)
        X, cells, mask = m.X, m.cells, m.dirichlet
    else:
        X, cells, mask = patch(*mesh)
        assert len(X) == mesh[0] * mesh[1]
    N = len(X)
    assert N <= 512
    g = BEMProblem(X, cells, mask, precision=PREC_MIXED, solver=SOLVER_LU)
    g.assemble_system()
    S, LU, _ = g.lu_factors()
    nblk = -(-N // B)
    P = nblk * B
    A, G = np.eye(P, dtype=f4), np.eye(P, dtype=f4)
    A[:N, :N], G[:N, :N] = S, LU
    invL, invU, late = [], [], None
    for b in range(nblk):
        d, r = slice(b * B, (b + 1) * B), slice((b + 1) * B, P)
        L, U, IL, cands = eliminate(A[d, d], G[d, d])
        assert np.array_equal(np.tril(L, -1) + U, G[d, d]), f"diagonal block {b}"
        invL.append(IL)
        if b + 1 < nblk:
            IU, _ = inv_u(U, cands, A[r, d], G[r, d])
            invU.append(IU)
            W = chain(IL, A[d, r])
            assert np.array_equal(W[:, :N - (b + 1) * B], G[d, r][:, :N - (b + 1) * B]), f"row panel {b}"
            A[r, r] -= chain(G[r, d], G[d, r])
        else:
            late = U, cands
    v = np.random.default_rng(3).normal(size=N)
    x = np.zeros(P, f4)
    x[:N] = v
    up, down = list(range(nblk)), list(range(nblk))[::-1]
    # forward, then the last block's reciprocals from the GPU's answer, bottom up
    y = sweep(G, invL, x, up, True)
    z = g.lu_apply(v)
    U, cands = late
    dinv, IU = np.array([c[0] for c in cands], f4), np.zeros((B, B), f4)
    for i in range(B - 1, -1, -1):
        for c in cands[i]:
            dinv[i] = c
            IU[i] = inv_u_row(U, i, dinv)
            o = (nblk - 1) * B + i
            if o >= N or diag_dot(IU[i:i + 1], y[(nblk - 1) * B:])[0] == z[o]:
                break
    invU.append(IU)
    assert np.array_equal(sweep(G, invU, y, down, True)[:N], z[:N].astype(f4)), "L, U"
    yt = sweep(G.T.copy(), [i.T.copy() for i in invU], x, up, False)
    zt = sweep(G.T.copy(), [i.T.copy() for i in invL], yt, down, False)
    assert np.array_equal(zt[:N], g.lu_apply(v, transpose=True).astype(f4)), "transposed"
