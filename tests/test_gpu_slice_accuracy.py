"""The FP64 rank updates by integer slices where the lines of a block's panels
hold entries of very different sizes: columns of A that are large and zero (or
absent) in part of a block's rows, and infinities.  A plain
elimination loses nothing there: its error does not change when a column is
multiplied by a power of two.

The systems are dense, with no interchange (diagonals of about ten times the
largest other entry), and set up in elimination order.  Tolerance: four times
the error of the oracle's plain FP64 elimination, both against the same
elimination in extended precision (numpy's longdouble), column by column
relative to the column's largest entry, L and U apart, and for the solution.
"""
import numpy as np
import pytest
import scipy.sparse as sp

import oracle
import sparspak as S
from sparspak.sparse_solver import _factor_, _inmatrix_, _matrix_arrays

pytestmark = pytest.mark.gpu


def solver(n):
    """A solver with a full n x n pattern, and its elimination order."""
    s = S.SparseSolver(sp.csc_matrix(np.ones((n, n))))
    S.findorder_(s)
    S.symbolicfactor_(s)
    return s, s.slvr.order.rperm - 1


def in_order(M, p):
    """The CSC matrix (every entry stored) that is eliminated as M."""
    A = np.empty_like(M)
    A[np.ix_(p, p)] = M
    full = sp.csc_matrix(np.ones(M.shape))
    full.data = A.ravel(order="F").copy()
    return full


def values(kind, n, power, seed=0):
    t = np.random.default_rng(seed)
    M = t.standard_normal((n, n)) + 0.15 * n * np.eye(n)
    big = np.ones(n)
    if kind == "above":        # zero in most rows of the first block
        M[:50, 150] = 0.0
    elif kind == "two":        # nonzero in one row of the first block, and on the diagonal
        M[:32, 150] = 0.0
        M[33:150, 150] = 0.0
        M[151:, 150] = 0.0
    elif kind == "several":
        for j, r in ((90, 17), (150, 50), (151, 63), (220, 5), (299, 40)):
            M[:r, j] = 0.0
            big[j] = 2.0 ** power
    if kind in ("above", "two"):
        big[150] = 2.0 ** power
    return M * big, big


def eliminate(M):
    M = M.astype(np.longdouble)
    for k in range(len(M) - 1):
        M[k + 1:, k] /= M[k, k]
        M[k + 1:, k + 1:] -= np.outer(M[k + 1:, k], M[k, k + 1:])
    return M


def dense_factor(slvr, lnz, unz):
    """L (below the diagonal) and U of the full pattern from the reference's layout."""
    n = slvr.n
    F = np.zeros((n, n))
    xs = slvr.xsuper - 1
    for j in range(n):
        k = slvr.snode[j] - 1
        F[xs[k]:, j] = lnz[slvr.xlnz[j] - 1: slvr.xlnz[j + 1] - 1]
        F[j, xs[k + 1]:] = unz[slvr.xunz[j] - 1: slvr.xunz[j + 1] - 1]
    return F


def errors(F, T):
    out = []
    for part in (np.triu, lambda X: np.tril(X, -1)):
        e, big = np.max(np.abs(part(F - T)), axis=0), np.max(np.abs(part(T)), axis=0)
        out.append(float(np.max(e[big > 0] / big[big > 0])))
    return out


@pytest.mark.parametrize("power", [0, 20, 40, 60])
@pytest.mark.parametrize("kind", ["above", "two", "several"])
def test_large_columns(kind, power):
    n = 300
    s, p = solver(n)
    M, big = values(kind, n, power)
    A = in_order(M, p)
    _inmatrix_(s.slvr, A)
    s.slvr.engine.profile_reset()
    _factor_(s.slvr)
    assert s.slvr.engine.profile_read()["tc_trail"]["launches"] > 0
    o = oracle.OracleLU(s.slvr)
    o.inmatrix_csc(*_matrix_arrays(A))
    assert o.factor() == 0
    assert np.array_equal(s.slvr.ipiv, o.ipiv)
    T = eliminate(M)
    F, G = (dense_factor(s.slvr, f.lnz, f.unz) for f in (s.slvr, o))
    ours, plain = errors(F, T), errors(G, T)
    b = np.random.default_rng(5).standard_normal(n)
    y = b.astype(np.longdouble)
    for i in range(n):
        y[i] -= T[i, :i] @ y[:i]
    for i in reversed(range(n)):
        y[i] = (y[i] - T[i, i + 1:] @ y[i + 1:]) / T[i, i]
    rhs = np.empty(n)
    rhs[p] = b
    for v, out in ((s.slvr.engine.solve(rhs.copy()), ours), (o.solve(rhs), plain)):
        out.append(float(np.max(np.abs(v.ravel()[p] - y) * big) / np.max(np.abs(y) * big)))   # columns' scale taken out
    print(kind, power, ours, plain)
    assert all(a <= 4.0 * max(b, 2.0 ** -52) for a, b in zip(ours, plain))


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_finite_columns_beside_a_non_finite_entry(bad):
    # small multipliers: an update that is dropped for the infinity's sake shows in the other columns.  Every entry is a
    # sum of at most n products that are 2^-30 of it, so that n u bounds its relative error
    n = 200
    s, p = solver(n)
    M = np.random.default_rng(1).uniform(0.5, 1.0, (n, n)) * 2.0 ** -30
    np.fill_diagonal(M, 1.0)
    M[40, 150] = bad
    A = in_order(M, p)
    _inmatrix_(s.slvr, A)
    _factor_(s.slvr)
    o = oracle.OracleLU(s.slvr)
    o.inmatrix_csc(*_matrix_arrays(A))
    o.factor()
    F, G = (dense_factor(s.slvr, f.lnz, f.unz) for f in (s.slvr, o))
    assert np.all(np.isfinite(F[:150, :150])) and np.all(np.isfinite(G[:150, :150]))
    both = np.isfinite(F) & np.isfinite(G)
    assert np.max(np.abs(F[both] / G[both] - 1.0)) <= n * 2.0 ** -53


@pytest.mark.parametrize("spd", [False, True])
@pytest.mark.parametrize("power", [20, 40])
def test_large_columns_of_a_grid(power, spd):
    # Schur complements over several blocks: some unknowns of a 3-D grid in other units (rows and columns in the
    # symmetric form), against the oracle's solution in the old ones; 1e-12 is the accuracy asked of plain FP64 solves
    # of these grids (condition number below 1e3)
    k = 16
    A = S.gallery.laplacian((k, k, k), shift=1e-3) if spd else S.gallery.convection_diffusion(k=k)
    n = A.shape[0]
    big = np.ones(n)
    big[np.random.default_rng(3).choice(n, 40, replace=False)] = 2.0 ** power
    B = sp.csc_matrix(A)
    B.data = B.data * np.repeat(big, np.diff(B.indptr)) * (big[B.indices] if spd else 1.0)
    s = S.SparseSolver(B, spd=spd)
    S.findorder_(s, S.nd_grid(k, k, k))
    S.symbolicfactor_(s)
    S.inmatrix_(s)
    s.slvr.engine.profile_reset()
    S.factor_(s)
    assert s.slvr.engine.profile_read()["tc_schur"]["launches"] > 0
    o = oracle.OracleLU(s.slvr)
    o.inmatrix_csc(*_matrix_arrays(sp.csc_matrix(A)))   # in the units it was in
    assert o.factor() == 0
    b = S.gallery.random_rhs(n, 1, seed=2).ravel()
    x = s.slvr.engine.solve(b * (big if spd else 1.0), "fp64+spd" if spd else "fp64").ravel() * big
    ref = o.solve(b).ravel()
    assert np.max(np.abs(x - ref)) <= 1e-12 * np.max(np.abs(ref))
