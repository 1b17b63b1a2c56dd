"""Rows below a small front's pivot block are scaled by the correctly rounded
reciprocal of the pivot, whichever way the front is factored: many one-column
fronts below a small dense root, whose L entries are one product each, so that
they are known to the bit."""
import numpy as np
import pytest
import scipy.sparse as sp

import sparspak as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("root", [2, 5, 17])
def test_l21_of_one_column_fronts(root, precision):
    leaves = 600
    n = leaves + root
    t = np.random.default_rng(root)
    A = np.zeros((n, n))
    A[leaves:, leaves:] = t.standard_normal((root, root)) + 4.0 * n * np.eye(root)
    A[:leaves, leaves:] = t.uniform(0.5, 1.0, (leaves, root))
    A[leaves:, :leaves] = t.uniform(0.5, 1.0, (root, leaves))
    A[np.arange(leaves), np.arange(leaves)] = t.uniform(1.0, 2.0, leaves)
    s = S.SparseSolver(sp.csc_matrix(A), precision=precision)
    S.findorder_(s)
    S.symbolicfactor_(s)
    S.inmatrix_(s)
    S.factor_(s)
    f = np.float32 if precision == "fp32" else np.float64
    p, x, lnz = s.slvr.order.rperm - 1, s.slvr.xlnz - 1, s.slvr.lnz
    checked = 0
    for j in np.flatnonzero(p < leaves)[:leaves - 2]:   # the last leaf is in the root's front
        if x[j + 1] - x[j] != 1 + root:
            continue
        rows = s.slvr.lindx[s.slvr.xlindx[s.slvr.snode[j] - 1] - 1:][1:1 + root] - 1   # in elimination order
        want = f(A[p[rows], p[j]]) * (f(1.0) / f(A[p[j], p[j]]))
        assert np.array_equal(lnz[x[j] + 1: x[j + 1]], want.astype(np.float64)), j
        checked += 1
    assert checked > leaves // 2
