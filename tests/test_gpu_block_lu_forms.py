"""The FP32 block LU where its pivots tie, are zero or NaN, or have reciprocals
outside the normal range, in every group of a block: identical pivots to the
oracle's, factors equal to the bit (ties: arithmetic on powers of two) or
within FP32 rounding, column by column (n u times an elimination growth below 4
for the diagonally dominant matrices, as in the tests of the block LU)."""
import numpy as np
import pytest
import scipy.sparse as sp
from scipy.linalg import hadamard

import oracle
from sparspak.sparse_solver import _factor_, _inmatrix_, _matrix_arrays
import sparspak as S

pytestmark = pytest.mark.gpu


def solver(n, maxblocksize, **kw):
    s = S.SparseSolver(sp.csc_matrix(np.ones((n, n))), precision="fp32", maxblocksize=maxblocksize, **kw)
    S.findorder_(s)
    S.symbolicfactor_(s)
    return s, s.slvr.order.rperm - 1


def factors(s, p, M):
    A = np.empty_like(M)
    A[np.ix_(p, p)] = M
    full = sp.csc_matrix(np.ones(M.shape))
    full.data = A.ravel(order="F").copy()
    _inmatrix_(s.slvr, full)
    o = oracle.OracleLU(s.slvr)
    o.inmatrix_csc(*_matrix_arrays(full))
    o.factor()
    _factor_(s.slvr)
    return o


@pytest.mark.parametrize("n", [40, 128, 200, 300])
@pytest.mark.parametrize("maxblocksize", [7, 30, 48])
def test_ties_in_every_group(n, maxblocksize):
    s, p = solver(n, maxblocksize)
    M = np.zeros((n, n))
    t = np.random.default_rng(n)
    xs = s.slvr.xsuper - 1
    for a, e in zip(xs[:-1], xs[1:]):   # Hadamard matrices, rows in random order, in the pieces
        k = 1 << int(np.log2(e - a))
        M[a:a + k, a:a + k] = hadamard(k)[t.permutation(k)]
        M[range(a + k, e), range(a + k, e)] = 1.0
    o = factors(s, p, M)
    assert np.array_equal(s.slvr.ipiv, o.ipiv)
    assert np.array_equal(s.slvr.lnz, o.lnz)


def large(n):
    """Factors that bring some of the diagonal entries of 2 n above 2^126."""
    big = np.ones(n)
    big[::9] = 2.0 ** (127 - np.floor(np.log2(2.0 * n)))
    return big


@pytest.mark.parametrize("n", [40, 128, 200])
def test_reciprocals_outside_the_normal_range(n):
    s, p = solver(n, 30)
    M = np.random.default_rng(n).standard_normal((n, n)) + 2.0 * n * np.eye(n)
    o = factors(s, p, M * large(n))
    assert np.array_equal(s.slvr.ipiv, o.ipiv)
    x = s.slvr.xlnz[:-1] - 1
    assert np.all(np.maximum.reduceat(np.abs(s.slvr.lnz - o.lnz), x) <= 5e-5 * np.maximum.reduceat(np.abs(o.lnz), x))


@pytest.mark.parametrize("n", [40, 128, 200])
def test_reciprocals_outside_the_normal_range_spd(n):
    s, p = solver(n, 30, spd=True)
    M = np.random.default_rng(n).standard_normal((n, n))
    M = np.tril(M) + np.tril(M, -1).T
    np.fill_diagonal(M, 2.0 * n * large(n))
    factors(s, p, M)
    C = np.linalg.cholesky(M)
    for j in range(n):
        f = int(s.slvr.xsuper[s.slvr.snode[j] - 1]) - 1
        got = s.slvr.lnz[s.slvr.xlnz[j] - 1: s.slvr.xlnz[j + 1] - 1][j - f:]
        assert np.max(np.abs(got - C[j:, j])) <= 5e-5 * np.max(np.abs(C[j:, j]))


@pytest.mark.parametrize("n", [40, 128])   # one block: the panels spread a NaN through their padded triangles
def test_nan(n):
    s, p = solver(n, 30)
    M = np.random.default_rng(n).standard_normal((n, n)) + 2.0 * n * np.eye(n)
    M[5, n // 2] = np.nan
    o = factors(s, p, M)
    end = int(s.slvr.xlnz[n // 2] - 1)   # the columns before it
    a, r = s.slvr.lnz[:end], o.lnz[:end]
    assert np.array_equal(s.slvr.ipiv[:n // 2], o.ipiv[:n // 2])
    assert np.all(np.isfinite(r)) and np.max(np.abs(a - r)) <= 5e-5 * np.max(np.abs(r))
    assert not np.any(np.isfinite(s.slvr.lnz) & ~np.isfinite(o.lnz))
