"""The FP64 rank updates on the tensor cores (integer slices) against the
oracle's plain FP64 elimination: dense systems of several blocks and a 3-D
grid (Schur complements), as they come and with rows, columns or both scaled
by random powers of two over 2^-60 .. 2^60, the symmetric form, and NaN.

Tolerance: eight times what separates two plain FP64 eliminations: the oracle's
factors of A and of A changed by n u entry by entry (u = 2^-53), and, for the
dense systems, the oracle's (left-looking, by supernodes) and a right-looking
one, column by column.  With rows scaled, pivots limited to a piece let the
errors grow, by how much the latter shows.
"""
import numpy as np
import pytest
import scipy.sparse as sp

import oracle
import sparspak as S

pytestmark = pytest.mark.gpu


def scales(n, how, seed):
    t = np.random.default_rng(seed)
    two = lambda: 2.0 ** t.integers(-60, 61, n)
    one = np.ones(n)
    if how == "both":
        d = two()
        return d, d
    return (two() if how == "rows" else one), (two() if how == "columns" else one)


def system(kind, how, seed=0):
    t = np.random.default_rng(seed)
    if kind == "grid":
        A = S.gallery.convection_diffusion(k=14)
        A.data *= t.uniform(0.9, 1.1, A.nnz)
        order = S.nd_grid(14, 14, 14)
    else:
        n = {"dense200": 200, "dense333": 333}[kind]
        A, order = sp.csc_matrix(t.standard_normal((n, n)) + 2.0 * n * np.eye(n)), None
    r, c = scales(A.shape[0], how, seed + 1)
    return sp.csc_matrix(sp.diags(r) @ A @ sp.diags(c)), order


def solver(A, order, **kw):
    s = S.SparseSolver(A, **kw)
    S.findorder_(s, order)
    S.symbolicfactor_(s)
    S.inmatrix_(s)
    return s


def oracle_of(s, A):
    o = oracle.OracleLU(s.slvr)
    o.inmatrix_csc(*S.sparse_solver._matrix_arrays(A))
    o.factor()
    return o


def right_looking(s, A, o):
    """lnz of the same elimination, one column after the other in FP64 with the oracle's pivots."""
    p = s.slvr.order.rperm - 1
    M = A.toarray()[np.ix_(p, p)]
    n, xs = M.shape[0], s.slvr.xsuper - 1
    for a, e in zip(xs[:-1], xs[1:]):
        for k in range(a, e):
            r = a + int(o.ipiv[k]) - 1
            M[[k, r], a:] = M[[r, k], a:]
            M[k + 1:, k] /= M[k, k]
            M[k + 1:, k + 1:] -= np.outer(M[k + 1:, k], M[k, k + 1:])
    out = np.empty(s.slvr.xlnz[-1] - 1)
    for j in range(n):
        f = xs[s.slvr.snode[j] - 1]
        out[s.slvr.xlnz[j] - 1: s.slvr.xlnz[j + 1] - 1] = M[f:, j]
    return out


def column_max(s, v):
    x = s.slvr.xlnz
    return np.maximum.reduceat(np.abs(v), x[:-1] - 1)


@pytest.mark.parametrize("how", ["none", "rows", "columns", "both"])
@pytest.mark.parametrize("kind", ["dense200", "dense333", "grid"])
def test_factors_vs_oracle(kind, how):
    A, order = system(kind, how)
    s = solver(A, order)
    eng = s.slvr.engine
    eng.profile_reset()
    S.factor_(s)
    prof = eng.profile_read()
    assert prof["tc_trail"]["launches"] > 0
    assert kind != "grid" or prof["tc_schur"]["launches"] > 0
    o = oracle_of(s, A)
    assert np.array_equal(s.slvr.ipiv, o.ipiv)
    P = A.copy()
    P.data *= 1.0 + A.shape[0] * 2.0 ** -53 * np.random.default_rng(2).uniform(-1.0, 1.0, P.nnz)
    q = oracle_of(s, P)
    assert np.array_equal(q.ipiv, o.ipiv)
    other = np.abs(q.lnz - o.lnz)
    if kind != "grid":
        other = np.maximum(other, np.abs(right_looking(s, A, o) - o.lnz))
    # lnz holds columns of L below the diagonal and of U above it, of very different sizes when scaled: entry by entry
    # against the column's largest, L and U apart
    for half in ("L", "U"):
        col = np.repeat(np.arange(A.shape[0]), np.diff(s.slvr.xlnz))
        first = np.repeat(s.slvr.xlnz[:-1] - 1, np.diff(s.slvr.xlnz))
        inpiece = col - (s.slvr.xsuper[s.slvr.snode[col] - 1] - 1)   # position of the diagonal in the column
        isU = np.arange(col.size) - first <= inpiece
        m = isU if half == "U" else ~isU
        err, per, ref = (np.where(m, np.abs(v), 0.0) for v in (s.slvr.lnz - o.lnz, other, o.lnz))
        e, d, big = (column_max(s, v) for v in (err, per, ref))
        ok = big > 0
        assert np.max(e[ok] / big[ok]) <= 8.0 * np.max(d[ok] / big[ok])


@pytest.mark.parametrize("how", ["none", "both"])
def test_symmetric_form(how):
    t = np.random.default_rng(3)
    n = 300
    M = t.standard_normal((n, n))
    r, _ = scales(n, how, 4)
    A = sp.csc_matrix(r[:, None] * (M @ M.T / n + np.eye(n)) * r)
    s = solver(A, None, spd=True)
    S.factor_(s)
    b = S.gallery.random_rhs(n, 3, seed=5) * r[:, None]
    x = np.array(b, order="F")
    S.triangularsolve_(s, x)
    ref = np.linalg.solve(M @ M.T / n + np.eye(n), b / r[:, None]) / r[:, None]
    # condition number below 10: 10 n u
    assert np.max(np.abs((x - ref) * r[:, None])) <= 10 * n * 2.0 ** -53 * np.max(np.abs(ref * r[:, None]))


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite(bad):
    A, _ = system("dense200", "none")
    A[3, 150] = bad
    s = solver(A, None)
    S.factor_(s)
    o = oracle_of(s, A)
    # nothing is finite where the oracle's is not (a plain FP64 update of padded triangles also spreads a NaN further)
    assert not np.any(np.isfinite(s.slvr.lnz) & ~np.isfinite(o.lnz))
