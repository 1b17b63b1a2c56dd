"""Memory of the FP64 slices (packed panels of the tensor-core rank updates):
allocated whenever the plan in use has them, in whatever order the options,
the values and the factorisation come, and refused without a trace.

Tolerance: 1e-10 against the oracle's solution and 1e-12 for the residual, as
the other solution tests on these grids.
"""
import numpy as np
import pytest

import oracle
import sparspak as S
from sparspak.sparse_solver import _ensure_engine, _inmatrix_, _matrix_arrays

pytestmark = pytest.mark.gpu

SIDE = 14   # a grid whose upper fronts take the slices


def system():
    A = S.gallery.convection_diffusion(k=SIDE)
    s = S.SparseSolver(A)
    S.findorder_(s, S.nd_grid(SIDE, SIDE, SIDE))
    S.symbolicfactor_(s)
    b = S.gallery.random_rhs(A.shape[0], 2, seed=1)
    return s, A, b


def check(s, A, b, x):
    o = oracle.OracleLU(s.slvr)
    o.inmatrix_csc(*_matrix_arrays(A))
    assert o.factor() == 0
    xo = o.solve(b)
    assert np.max(np.abs(x - xo)) <= 1e-10 * np.max(np.abs(xo))
    assert np.max(np.linalg.norm(b - A @ x, axis=0) / np.linalg.norm(b, axis=0)) <= 1e-12


def slices(eng):
    p = eng.profile_read()
    return p["tc_trail"]["launches"] + p["tc_schur"]["launches"] > 0


@pytest.mark.parametrize("fused", [False, True])
def test_option_switched_back_between_load_and_factor(fused):
    # the values' first assembly is under a plan without slices, their factorisation under one with them
    s, A, b = system()
    eng = _ensure_engine(s.slvr)
    eng.set_option("lu_pieces", 1)
    _inmatrix_(s.slvr, A)
    eng.set_option("lu_pieces", 0)
    eng.profile_reset()
    x = np.zeros_like(b, order="F")
    if fused:
        eng.factor_refine(b, x, "fp64")
    else:
        eng.factor("fp64")
        x = eng.solve(np.array(b, order="F"), "fp64")
    assert slices(eng)
    check(s, A, b, x)


def test_refused_slices():
    # a factorisation without them, one with them again, and solves captured under either plan
    s, A, b = system()
    eng = _ensure_engine(s.slvr)
    for limit in (-1, 0, 4096, -1):
        eng.set_option("slice_limit", limit)
        assert eng.get_option("slice_limit") == limit
        _inmatrix_(s.slvr, A)
        eng.profile_reset()
        eng.factor("fp64")
        assert slices(eng) == (limit < 0)
        for _ in range(2):   # captured, then replayed
            check(s, A, b, eng.solve(np.array(b, order="F"), "fp64"))


def test_solve_captured_before_a_refusal():
    # factored without slices by the option, solved (captured) under a plan that has them, then loaded again where
    # they are refused: the replayed solve must not belong to the plan that was dropped
    s, A, b = system()
    eng = _ensure_engine(s.slvr)
    eng.set_option("slice_limit", 0)
    eng.set_option("lu_pieces", 1)
    _inmatrix_(s.slvr, A)
    eng.factor("fp64")
    eng.set_option("lu_pieces", 0)
    check(s, A, b, eng.solve(np.array(b, order="F"), "fp64"))
    _inmatrix_(s.slvr, A)   # the slices are refused here
    eng.factor("fp64")
    assert not slices(eng)
    check(s, A, b, eng.solve(np.array(b, order="F"), "fp64"))


def test_slices_make_room():
    # an allocation that finds no memory gets that of the slices first; here not even that is enough, the call fails
    # with a status, and the factor and the next factorisations are sound
    import ctypes

    from sparspak import _native as N

    s, A, b = system()
    eng = _ensure_engine(s.slvr)
    _inmatrix_(s.slvr, A)
    eng.profile_reset()
    eng.factor("fp64")
    assert slices(eng)
    rc = N.gpu().spk_solve(eng._h, ctypes.c_void_p(1), 1 << 40, A.shape[0], N.SPK_HOST, N.SPK_FP64)   # the right-hand sides are not read
    assert rc == N.SPK_ENOMEM
    check(s, A, b, eng.solve(np.array(b, order="F"), "fp64"))
    for fused in (False, True):
        _inmatrix_(s.slvr, A)
        x = np.zeros_like(b, order="F")
        eng.profile_reset()
        if fused:
            eng.factor_refine(b, x, "fp64")
        else:
            eng.factor("fp64")
            x = eng.solve(np.array(b, order="F"), "fp64")
        assert slices(eng)   # there is room again
        check(s, A, b, x)


def test_pack_of_one_level_serves_all():
    # levels use the same memory for their slices: a system with tensor-core fronts on several levels, every factor
    # entry against the oracle's
    k = 20
    A = S.gallery.convection_diffusion(k=k)
    s = S.SparseSolver(A)
    S.findorder_(s, S.nd_grid(k, k, k))
    S.symbolicfactor_(s)
    _inmatrix_(s.slvr, A)
    eng = s.slvr.engine
    eng.profile_reset()
    S.sparse_solver._factor_(s.slvr)
    assert eng.profile_read()["tc_schur"]["launches"] >= 2
    o = oracle.OracleLU(s.slvr)
    o.inmatrix_csc(*_matrix_arrays(A))
    assert o.factor() == 0
    assert np.array_equal(s.slvr.ipiv, o.ipiv)
    for a, r in ((s.slvr.lnz, o.lnz), (s.slvr.unz, o.unz[: s.slvr.unz.size])):
        assert np.max(np.abs(a - r)) <= 1e-12 * np.max(np.abs(r))
