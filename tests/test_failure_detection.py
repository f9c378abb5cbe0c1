"""Failure detection and the reference's error contract, with every failure
made on the host or by a device wait given too little time -- nothing here
faults, traps or hangs a GPU:

* a device-side wait that runs out (the pipelined solves' block flags, the
  tensor-core Schur update's copy/MMA barriers; symla_gpu_set_wait_limit_ns)
  returns SYMLA_ERR_TIMEOUT, and the context stays usable;
* a context whose plan exceeds its device-memory limit fails with
  SYMLA_ERR_OOM (symla_gpu_set_memory_limit), and the next one succeeds;
* NaN / Inf injected into the matrix values: the calls return, and the same
  context factorizes the clean values correctly afterwards;
* size and call-order errors map to the reference's exceptions with its
  messages (solver.hpp:54-55, :140-143, :198-209, :299-315, :403-413).
"""
import ctypes as C

import numpy as np
import pytest

from ma57_b200 import (InvalidArgument, LogicError, Mode, OrderingType, Precision, RefinementOptions, SymLDLT)
from ma57_b200 import _lib as L
from ma57_b200 import matrices as M
from ma57_b200.solver import as_csc


def backward_error(A, X, B):
    R = B - M.sym_full(A) @ X
    normA = abs(A).sum(axis=1).max()
    return np.abs(R).max() / (normA * np.abs(X).max() + np.abs(B).max())


def test_kkt_block_size_errors_on_host():
    """setKKTBlockSizes rejects negative sizes (solver.hpp:54-55)."""
    s = SymLDLT()
    with pytest.raises(InvalidArgument, match="sizes must be nonnegative"):
        s.setKKTBlockSizes(-1, 3)


def test_factorize_before_analyze_is_a_logic_error():
    """solver.hpp:140-143."""
    A, _ = M.config1(4)
    with pytest.raises(LogicError, match="analyzePattern must be called first"):
        SymLDLT().factorize(A)


def test_memory_limit_rejects_negative():
    lib = L.load()
    assert lib.symla_gpu_set_memory_limit(-5) == L.SYMLA_ERR_INVALID
    assert lib.symla_gpu_set_memory_limit(0) == L.SYMLA_OK


@pytest.mark.gpu
def test_solve_wait_timeout_is_reported_and_context_survives():
    """A 1 ns limit cannot cover the forward solve's chain of 64-row blocks
    (each waits for the one before it), so a wait runs out: the solve
    returns SYMLA_ERR_TIMEOUT. With the default limit the same context solves
    again, bit for bit as before."""
    A, B = M.config3(24, nrhs=4)
    s = SymLDLT()
    s.setOrdering(OrderingType.Metis)
    s.analyzePattern(A)
    s.factorize(A)
    assert s.plan_stats()["max_m"] > 256  # fronts with several row blocks
    X0 = s.solve(B)
    lib = L.load()
    assert lib.symla_gpu_set_wait_limit_ns(s._ctx.h, 1) == L.SYMLA_OK
    with pytest.raises(RuntimeError, match="timed out") as ei:
        s.solve(B)
    assert "status 7" in str(ei.value)  # SYMLA_ERR_TIMEOUT
    assert lib.symla_gpu_set_wait_limit_ns(s._ctx.h, 0) == L.SYMLA_OK
    X1 = s.solve(B)
    np.testing.assert_array_equal(X1, X0)
    assert backward_error(A, X1, B) < 1e-12


@pytest.mark.gpu
def test_lowered_wait_limit_does_not_count_the_tree():
    """A band matrix in its natural order: a chain of 1500 fronts of one row
    block each, so that no block waits for another of its front. The solve takes
    milliseconds, far longer than the limit, which bounds the waits inside a
    front and not a front's wait for everything below it in the tree."""
    import scipy.sparse as sp
    from ma57_b200.solver import SymbolicFactorOptions
    n, band = 1500, 40
    st = M.Stream(3)
    A = sp.diags([st.uniform(n - d, -1.0, 1.0) for d in range(1, band + 1)], [-d for d in range(1, band + 1)])
    A = M.lower(sp.csc_matrix(A + sp.diags(np.where(np.arange(n) % 2 == 0, 100.0, -100.0))))
    B = np.asfortranarray(M.Stream(4).normal(2 * n).reshape(n, 2))
    s = SymLDLT()
    s.setOrdering(OrderingType.Natural)
    s.analyzePattern(A, SymbolicFactorOptions(0, 0.0))
    s.factorize(A)
    assert s.plan_stats()["levels"] > 1000 and 32 < s.plan_stats()["max_m"] <= 64
    X0 = s.solve(B)
    lib = L.load()
    assert lib.symla_gpu_set_wait_limit_ns(s._ctx.h, 20000) == L.SYMLA_OK
    np.testing.assert_array_equal(s.solve(B), X0)
    assert lib.symla_gpu_set_wait_limit_ns(s._ctx.h, 0) == L.SYMLA_OK
    np.testing.assert_array_equal(s.solve(B), X0)
    assert backward_error(A, X0, B) < 1e-12


@pytest.mark.gpu
def test_tensor_core_wait_timeout_is_reported_and_context_survives():
    """The mixed-precision far update waits on TMA copies and MMA groups; a
    1 ns limit makes those waits run out. The CTA abandons its tile, drains
    (within the default limit) what it has in flight and frees its tensor
    memory; the factorization returns SYMLA_ERR_TIMEOUT. With the default
    limit the same context factorizes to the right inertia."""
    A, B = M.config3(24, nrhs=2)
    s = SymLDLT()
    s.setOrdering(OrderingType.Metis)
    s.setPrecision(Precision.Mixed)
    s.analyzePattern(A)
    s.factorize(A)
    good = s.inertia().as_tuple()
    lib = L.load()
    lib.symla_gpu_reset_kernel_stats(s._ctx.h)
    assert lib.symla_gpu_set_wait_limit_ns(s._ctx.h, 1) == L.SYMLA_OK
    with pytest.raises(RuntimeError, match="timed out") as ei:
        s.factorize(A)
    assert "status 7" in str(ei.value)
    assert "no longer usable" not in str(ei.value)
    with pytest.raises(LogicError):  # the failed factorization is not solvable
        s.solve(B)
    assert lib.symla_gpu_set_wait_limit_ns(s._ctx.h, 0) == L.SYMLA_OK
    s.factorize(A)
    assert s.inertia().as_tuple() == good
    r = s.solveWithRefinement(A, B, RefinementOptions(tolerance=1e-12))
    assert r.diagnostics.final_relative_residual <= 1e-12


@pytest.mark.gpu
def test_undersized_memory_limit_gives_oom_then_recovers():
    """A plan that does not fit the device-memory limit fails with
    SYMLA_ERR_OOM at create time (no context is returned); with the limit
    lifted the same analysis creates and factorizes."""
    A, b = M.config1(12)
    s = SymLDLT()
    s.analyzePattern(A)
    lib = L.load()
    _, cp, ri, _ = as_csc(A)
    try:
        assert lib.symla_gpu_set_memory_limit(64 * 1024) == L.SYMLA_OK
        h = C.c_void_p()
        rc = lib.symla_gpu_create(s._analysis.h, A.shape[0], L.ptr_i(cp), L.ptr_i(ri), 0, C.byref(h))
        assert rc == L.SYMLA_ERR_OOM
        assert not h.value
        assert "memory limit" in L.last_error()
        with pytest.raises(RuntimeError, match="memory limit"):
            s.factorize(A)
    finally:
        lib.symla_gpu_set_memory_limit(0)
    s.factorize(A)
    assert s.inertia().as_tuple() == (1720 - 6, 6, 0) or sum(s.inertia().as_tuple()) == A.shape[0]
    x = s.solve(b)
    assert backward_error(A, x, b) < 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("precision", [Precision.FP64, Precision.Mixed])
def test_nonfinite_values_then_clean_refactorization(bad, precision):
    """Host-injected NaN / Inf in the values (the reference does not check
    for them either): factorize, solve and refinement return without hanging
    and without reporting a converged solution, and the same context then
    refactorizes the clean values to the right inertia and accuracy."""
    A, B = M.config3(20, nrhs=2)
    s = SymLDLT()
    s.setOrdering(OrderingType.Metis)
    s.setPrecision(precision)
    s.analyzePattern(A)
    s.factorize(A)
    good = s.inertia().as_tuple()
    Abad = A.copy()
    Abad.data[Abad.nnz // 2] = bad
    s.factorize(Abad)
    if not s.isSingular():
        r = s.solveWithRefinement(Abad, B, RefinementOptions(max_iterations=3, tolerance=1e-12))
        assert not (r.diagnostics.final_relative_residual <= 1e-12)
    else:
        with pytest.raises(LogicError, match="numerically singular"):
            s.solve(B)
    s.factorize(A)
    assert s.inertia().as_tuple() == good
    r = s.solveWithRefinement(A, B, RefinementOptions(tolerance=1e-12))
    assert r.diagnostics.final_relative_residual <= 1e-12
    assert backward_error(A, r.x, B) <= 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("ctas", [0, 1])
@pytest.mark.parametrize("n", [16, 32, 33, 128, 129, 300, 784, 800])
def test_nonfinite_pivots_are_not_perturbed(n, ctas, bad):
    """Static pivoting adds delta to a pivot that fails the floor test and
    counts that one: a NaN never fails it, nor does an infinite pivot of the
    expected sign. One front of each kernel's range (ctas = 1: the single-CTA
    panels), the bad entry on the last diagonal, so that every other pivot is
    finite and well above the floor."""
    import scipy.sparse as sp
    G = M.Stream(n).normal(n * n).reshape(n, n)
    K = (G + G.T) / 2 + 4 * n * np.eye(n)
    K[n - 1, n - 1] = bad
    A = M.lower(sp.csc_matrix(K))
    lib = L.load()
    s = SymLDLT()
    s.setOrdering(OrderingType.Natural)
    s.analyzePattern(A)
    _, cp, ri, vals = as_csc(A)
    h = s._context(cp, ri).h
    for lv in range(int(s.plan_stats()["levels"])):
        assert lib.symla_gpu_set_level_schedule(h, lv, 0, ctas) == L.SYMLA_OK
    o, info, signs = L.FactorOpts(), L.FactorInfo(), np.ones(n, np.int32)
    lib.symla_factor_opts_default(C.byref(o))
    o.mode = L.MODE_STATIC
    o.static_delta, o.static_rel_floor, o.static_abs_floor = 1.0, 0.0, 1e-300  # (a relative floor would be infinite)
    o.expected_sign = L.ptr_i(signs)
    assert lib.symla_gpu_factorize(h, L.ptr_d(vals), 0, C.byref(o), C.byref(info)) == L.SYMLA_OK
    assert info.num_perturbed == 0 and info.total_perturbation == 0.0
    assert info.n_pos == (n if bad == np.inf else n - 1)


@pytest.mark.gpu
@pytest.mark.parametrize("n,ctas", [(16, 0), (100, 0), (300, 1), (300, 2), (800, 1), (800, 16)])
def test_no_candidate_under_a_negative_zero_tolerance(n, ctas):
    """The last pivot has no other candidate; a negative zero tolerance does not
    take it for isolated, and a NaN fails every test against it: it is a 1x1
    pivot (in every kernel's range), not a search at row -1."""
    import scipy.sparse as sp
    G = M.Stream(n).normal(n * n).reshape(n, n)
    K = (G + G.T) / 2 + 4 * n * np.eye(n)
    K[n - 1, n - 1] = np.nan
    A = M.lower(sp.csc_matrix(K))
    lib = L.load()
    s = SymLDLT()
    s.setOrdering(OrderingType.Natural)
    s.analyzePattern(A)
    _, cp, ri, vals = as_csc(A)
    h = s._context(cp, ri).h
    for lv in range(int(s.plan_stats()["levels"])):
        assert lib.symla_gpu_set_level_schedule(h, lv, 0, ctas) == L.SYMLA_OK
    o, info = L.FactorOpts(), L.FactorInfo()
    lib.symla_factor_opts_default(C.byref(o))
    o.zero_tolerance = -1.0
    assert lib.symla_gpu_factorize(h, L.ptr_d(vals), 0, C.byref(o), C.byref(info)) == L.SYMLA_OK
    assert (info.n_pos, info.n_neg, info.n_zero, info.singular) == (n - 1, 0, 1, 0)


@pytest.mark.gpu
def test_size_and_order_errors_match_the_reference():
    A, b = M.config1(6)
    n = A.shape[0]
    s = SymLDLT()
    s.analyzePattern(A)
    with pytest.raises(LogicError, match=r"factorize\(\) must be called before solve\(\)"):
        s.solve(b)
    s.factorize(A)
    with pytest.raises(InvalidArgument, match="B.rows"):
        s.solve(np.ones(n + 1))
    lib = L.load()
    X = np.zeros(n)
    bb = np.ascontiguousarray(b)
    assert lib.symla_gpu_solve(s._ctx.h, L.ptr_d(bb), n, -1, L.ptr_d(X), n, 0) == L.SYMLA_ERR_BAD_SIZE
    assert lib.symla_gpu_solve(s._ctx.h, L.ptr_d(bb), n - 1, 1, L.ptr_d(X), n, 0) == L.SYMLA_ERR_BAD_SIZE
    assert lib.symla_gpu_solve(s._ctx.h, L.ptr_d(bb), n, 1, L.ptr_d(X), n - 1, 0) == L.SYMLA_ERR_BAD_SIZE
    # the context is untouched by rejected calls
    x = s.solve(b)
    assert backward_error(A, x, b) < 1e-12
    # StaticRegularized size checks (solver.hpp:299-315)
    k = SymLDLT()
    k.setMode(Mode.StaticRegularized)
    k.setKKTBlockSizes(n - 1, 2)
    k.analyzePattern(A)
    with pytest.raises(InvalidArgument, match="do not sum to the matrix size"):
        k.factorize(A)
    k.setExpectedSignPattern(np.ones(n - 3, np.int32))
    with pytest.raises(InvalidArgument, match="does not match the matrix size"):
        k.factorize(A)
    # retry budget exhausted (solver.hpp:403-413): the indefinite stencil
    # cannot have the all-positive inertia a one-block KKT expects
    k.setKKTBlockSizes(0, n)
    k.setMaxRegularizationRetries(0)
    with pytest.raises(RuntimeError, match="retry budget"):
        k.factorize(A)
