"""FP64 factors of a dense system whose columns differ by more than the exponent
range of a quotient: no entry of the factors over- or underflows, and a plain
elimination's error does not change when columns are multiplied by powers of
two.  Block LU, panels and updates in one and in several blocks.

Tolerance: four times the oracle's error, both against the elimination of the
unscaled system in extended precision, column by column, L and U apart.
"""
import numpy as np
import pytest

import oracle
from sparspak.sparse_solver import _factor_, _inmatrix_, _matrix_arrays
from test_gpu_slice_accuracy import dense_factor, eliminate, errors, in_order, solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [30, 60, 100, 200])
def test_columns_beyond_the_range_of_a_quotient(n):
    s, p = solver(n)
    M = np.random.default_rng(n).standard_normal((n, n)) + 0.15 * n * np.eye(n) + 8.0 * np.eye(n)
    big = np.ones(n)
    big[[3, n // 2]] = 2.0 ** -600
    big[[9, n // 3, n - 7]] = 2.0 ** 600
    A = in_order(M * big, p)
    _inmatrix_(s.slvr, A)
    _factor_(s.slvr)
    o = oracle.OracleLU(s.slvr)
    o.inmatrix_csc(*_matrix_arrays(A))
    assert o.factor() == 0
    assert np.array_equal(s.slvr.ipiv, o.ipiv)
    T = eliminate(M)
    take = np.triu(np.broadcast_to(1.0 / big, (n, n))) + np.tril(np.ones((n, n)), -1)   # L does not change with the columns
    F, G = (dense_factor(s.slvr, f.lnz, f.unz) * take for f in (s.slvr, o))
    ours, plain = errors(F, T), errors(G, T)
    print(n, ours, plain)
    assert np.all(np.isfinite(F))
    assert all(a <= 4.0 * max(b, 2.0 ** -52) for a, b in zip(ours, plain))
