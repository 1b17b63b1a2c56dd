"""The FP64 rank updates by integer slices beside infinities and NaN: what a
plain elimination leaves finite is right.  The system is dense, with no
interchange, and set up in elimination order.
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
