"""Groups of four right-hand sides side by side in the solves of large fronts:
one front of several blocks (FP32 in one cluster pass, FP64 in chunks), numbers
of right-hand sides around the groups and the 16 columns of a call.

Tolerance: a strictly diagonally dominant matrix by rows and columns is factored
without interchanges with | |L| |U| | <= 3 |A| (infinity norm), and
|b - A x| <= 3 n u | |L| |U| | |x|.
"""
import numpy as np
import pytest
import scipy.sparse as sp

import sparspak as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n", [500, 1100])
@pytest.mark.parametrize("nrhs", [1, 4, 5, 13, 16, 18])
def test_dense_front(n, nrhs, precision):
    rng = np.random.default_rng(n)
    A = rng.uniform(-1.0, 1.0, (n, n))
    np.fill_diagonal(A, n)
    s = S.SparseSolver(sp.csc_matrix(A), precision=precision)
    S.findorderperm_(s, np.arange(1, n + 1))
    S.symbolicfactor_(s)
    S.inmatrix_(s)
    S.factor_(s)
    b = S.gallery.random_rhs(n, nrhs, seed=nrhs).reshape(n, nrhs)
    u = 2.0 ** (-53 if precision == "fp64" else -24)
    for M, solve in ((A, S.triangularsolve_), (A.T, S.transposetriangularsolve_)):
        x = b.copy(order="F")
        solve(s, x)
        r = np.max(np.abs(b - M @ x), axis=0)
        bound = 9.0 * n * u * np.max(np.sum(np.abs(M), axis=1)) * np.max(np.abs(x), axis=0)
        assert np.all(r <= bound)
