"""Small fronts (factored and solved whole by a warp each) against the oracle
in FP64: banded systems, whose chains of small supernodes merge into fronts of
several width classes, with as many rows below them as the band is wide: the
rows below a block both in the warp that factors it and not, in-block
interchanges, and the symmetric form.

Tolerance: n u = 2e-14 for n = 200 times an element growth of at most 50.
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
        scale = np.max(np.abs(o.lnz))
        assert np.max(np.abs(s.slvr.lnz - o.lnz)) <= 1e-12 * scale
        assert np.max(np.abs(s.slvr.unz - o.unz[: s.slvr.unz.size])) <= 1e-12 * scale
    for transpose in (False, True):
        x = b.copy(order="F")
        (S.transposetriangularsolve_ if transpose else S.triangularsolve_)(s, x)
        M = A.T if transpose else A
        r = np.linalg.norm(b - M @ x, axis=0)
        # backward error with the growth above, against |A| |x| + |b|
        assert np.max(r / (sp.linalg.norm(A) * np.linalg.norm(x, axis=0) + np.linalg.norm(b, axis=0))) <= 1e-12
