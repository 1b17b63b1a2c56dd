"""The FP32 block LU on dense blocks against the oracle: identical pivots and
factors within FP32 rounding, at the edges of its 32-column groups and 128-
column blocks and in each of its forms (diagonal pivots throughout, pivots
that are searched for, ties, zero pivots, pieces wider than a group).

Tolerances: n u = 1.2e-5 for n = 200 times the growth of the elimination,
which is below 4 for the diagonally dominant matrices and, with pivots
limited to a piece, at most some hundreds for the others.
"""
import numpy as np
import pytest
import scipy.sparse as sp

import oracle
import sparspak as S

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.max(np.abs(a - b)) / np.max(np.abs(b)))


def dense(kind, n, seed=0):
    rng = np.random.default_rng(seed)
    M = rng.standard_normal((n, n))
    if kind == "dominant":
        return M + 2.0 * n * np.eye(n)
    M += 0.5 * np.sqrt(n) * np.eye(n)
    if kind == "ties":   # the first column, and one that starts a piece, of equal sizes
        M[:, 0] = np.sign(M[:, 0])
    return M


@pytest.mark.parametrize("n", [33, 64, 97, 128, 129, 200])
@pytest.mark.parametrize("kind", ["dominant", "pivoting", "ties"])
@pytest.mark.parametrize("maxblocksize", [30, 7, 48])
def test_dense_blocks(kind, n, maxblocksize):
    A = sp.csc_matrix(dense(kind, n))
    s = S.SparseSolver(A, precision="fp32", maxblocksize=maxblocksize)
    S.findorder_(s)
    S.symbolicfactor_(s)
    assert np.max(np.diff(s.slvr.xsuper)) <= 64
    o = oracle.OracleLU(s.slvr)
    o.inmatrix_csc(*S.sparse_solver._matrix_arrays(A))
    o.factor()
    S.inmatrix_(s)
    S.factor_(s)
    assert np.array_equal(s.slvr.ipiv, o.ipiv)
    assert rel(s.slvr.lnz, o.lnz) <= (5e-5 if kind == "dominant" else 5e-3)


@pytest.mark.parametrize("n", [40, 128, 150])
def test_zero_pivot(n):
    M = dense("dominant", n)
    M[:, n // 2] = 0.0
    s = S.SparseSolver(sp.csc_matrix(sp.coo_matrix(np.ones((n, n)))), precision="fp32")
    A = s.p.copy()
    A.data[:] = M.T.ravel()
    s.p = A
    S.findorder_(s)
    S.symbolicfactor_(s)
    S.inmatrix_(s)
    col = int(s.slvr.order.rinvp[n // 2])
    with pytest.raises(S.ErrorException, match=f"supernode {int(s.slvr.snode[col - 1])}\\."):
        S.factor_(s)


@pytest.mark.parametrize("n", [33, 100, 129])
def test_spd_blocks(n):
    M = dense("pivoting", n)
    A = sp.csc_matrix(M @ M.T / n + np.eye(n))
    s = S.SparseSolver(A, precision="fp32", spd=True)
    S.findorder_(s)
    S.symbolicfactor_(s)
    S.inmatrix_(s)
    S.factor_(s)
    p = s.slvr.order.rperm - 1
    C = np.linalg.cholesky(A.toarray()[np.ix_(p, p)])
    L = np.zeros((n, n))
    for j in range(n):
        f = int(s.slvr.xsuper[s.slvr.snode[j] - 1]) - 1
        L[f:, j] = s.slvr.lnz[s.slvr.xlnz[j] - 1: s.slvr.xlnz[j + 1] - 1]
    assert rel(np.tril(L), C) <= 5e-5


@pytest.mark.parametrize("n", [33, 63, 64, 65, 128, 150])
@pytest.mark.parametrize("kind", ["dominant", "pivoting", "ties"])
@pytest.mark.parametrize("maxblocksize", [30, 7, 48])
def test_dense_blocks_fp64(kind, n, maxblocksize):
    """FP64: eight times what a change of A by n u moves the oracle's factors by
    (the growth of the elimination is below 8 of it: pivots limited to a piece
    of at most 48 rows of matrices with a diagonal of sqrt(n) / 2)."""
    A = sp.csc_matrix(dense(kind, n))
    s = S.SparseSolver(A, maxblocksize=maxblocksize)
    S.findorder_(s)
    S.symbolicfactor_(s)
    P = A.copy()
    P.data *= 1.0 + n * 2.0 ** -53 * np.random.default_rng(1).uniform(-1.0, 1.0, P.nnz)
    if kind == "ties":   # the perturbed copy keeps them
        P[:, 0] = A[:, 0]
    o, q = (oracle.OracleLU(s.slvr) for _ in range(2))
    for orc, M in ((o, A), (q, sp.csc_matrix(P))):
        orc.inmatrix_csc(*S.sparse_solver._matrix_arrays(M))
        orc.factor()
    S.inmatrix_(s)
    S.factor_(s)
    assert np.array_equal(s.slvr.ipiv, o.ipiv) and np.array_equal(q.ipiv, o.ipiv)
    assert np.max(np.abs(s.slvr.lnz - o.lnz)) <= 8.0 * np.max(np.abs(q.lnz - o.lnz))
