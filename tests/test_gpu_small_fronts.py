"""Small fronts (factored and solved whole by a warp each) against the oracle
in FP64: banded systems, whose chains of small supernodes merge into fronts of
several width classes, with as many rows below them as the band is wide: the
rows below a block both in the warp that factors it and not, in-block
interchanges, and the symmetric form.

Tolerance: the factors of a backward stable elimination are those of a matrix
within n u g of A, entry by entry (u = 2^-53, g the growth of the elimination);
what such a change moves the oracle's factors by is measured with the oracle,
and four times that is allowed.
"""
import numpy as np
import pytest
import scipy.sparse as sp

import oracle
import sparspak as S

pytestmark = pytest.mark.gpu


def banded(n, band, kind, seed=0):
    rng = np.random.default_rng(seed)
    d = [rng.uniform(-1.0, 1.0, n - abs(k)) for k in range(-band, band + 1)]
    A = sp.diags(d, range(-band, band + 1), format="csc")
    if kind == "spd":
        A = A + A.T + 2.5 * (band + 1) * sp.identity(n)
    elif kind == "dominant":
        A = A + 1.5 * (band + 1) * sp.identity(n)
    else:   # interchanges inside the pieces
        A = A + 0.5 * np.sqrt(band + 1) * sp.identity(n)
    return sp.csc_matrix(A)


@pytest.mark.parametrize("kind", ["dominant", "pivoting", "spd"])
@pytest.mark.parametrize("n,band", [(5, 1), (33, 1), (200, 1), (200, 2), (200, 7), (130, 15), (130, 17), (130, 31), (130, 33)])
def test_banded(n, band, kind):
    A = banded(n, band, kind)
    s = S.SparseSolver(A, spd=kind == "spd")
    S.findorderperm_(s, np.arange(1, n + 1))
    S.symbolicfactor_(s)
    S.inmatrix_(s)
    S.factor_(s)
    b = S.gallery.random_rhs(n, 5, seed=1)
    if kind != "spd":
        o = oracle.OracleLU(s.slvr)
        o.inmatrix_csc(*S.sparse_solver._matrix_arrays(A))
        o.factor()
        assert np.array_equal(s.slvr.ipiv, o.ipiv)
        g = max(1.0, np.max(np.abs(o.lnz)) / np.max(np.abs(A.data)))
        P = A.copy()
        P.data *= 1.0 + n * 2.0 ** -53 * g * np.random.default_rng(2).uniform(-1.0, 1.0, P.nnz)
        q = oracle.OracleLU(s.slvr)
        q.inmatrix_csc(*S.sparse_solver._matrix_arrays(P))
        q.factor()
        assert np.array_equal(q.ipiv, o.ipiv)
        nu = s.slvr.unz.size
        assert np.max(np.abs(s.slvr.lnz - o.lnz)) <= 4.0 * np.max(np.abs(q.lnz - o.lnz))
        assert np.max(np.abs(s.slvr.unz - o.unz[:nu])) <= 4.0 * np.max(np.abs(q.unz[:nu] - o.unz[:nu]))
    for transpose in (False, True):
        x = b.copy(order="F")
        (S.transposetriangularsolve_ if transpose else S.triangularsolve_)(s, x)
        M = A.T if transpose else A
        r = np.linalg.norm(b - M @ x, axis=0)
        lu = np.max(np.abs(s.slvr.lnz)) * (1.0 if kind == "spd" else max(1.0, np.max(np.abs(s.slvr.lnz))))
        # |b - A x| <= 3 n u |L| |U| |x|, with |L| |U| from the largest entries over a band
        assert np.max(r / (lu * np.linalg.norm(x, axis=0))) <= 3.0 * n * 2.0 ** -53 * (2 * band + 1) * np.sqrt(n)
