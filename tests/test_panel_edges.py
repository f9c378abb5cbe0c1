"""Panels of large fronts (one dense front, natural order). Static pivoting at
the edges of the 32-pivot panels, the 96-row CTAs and the 256-pivot outer
blocks, against the CPU oracle: inertia, perturbed pivots and residual.
Threshold pivoting on both sides of the single-CTA panel's range."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

from ma57_b200 import Mode, OrderingType, SymLDLT
from ma57_b200 import _lib as L
from ma57_b200.matrices import Stream, lower
from oracle.pyoracle import OracleSymLDLT


def quasi_definite(n, n1, weak):
    """Dense [[-E, A^T], [A, F]] of n1 + (n - n1), rows interleaved; `weak`
    diagonal entries have the wrong sign and are perturbed."""
    st = Stream(1000 * n + n1)
    G = st.normal(n * n).reshape(n, n) / np.sqrt(n)
    K = G @ G.T + np.eye(n)
    sign = np.where((np.arange(n) * n1) % n < n1, -1, 1)
    S = np.outer(sign, sign)
    K = np.where(S > 0, K * sign[:, None], (G + G.T) / 4)
    for i in range(weak):
        j = (i * 37 + 5) % n
        K[j, j] = -1e-3 * sign[j]
    return K, sign


@pytest.mark.gpu
@pytest.mark.parametrize("n", [129, 160, 161, 225, 256, 257, 289, 545, 801])
@pytest.mark.parametrize("weak", [0, 3])
def test_static_dense_front(n, weak):
    K, sign = quasi_definite(n, n // 3, weak)
    A = lower(sp.csc_matrix(K))
    s = SymLDLT()
    s.setMode(Mode.StaticRegularized)
    s.setOrdering(OrderingType.Natural)
    s.setExpectedSignPattern(sign)
    s.setStaticPivotFloor(1e-8)
    s.setInitialRegularizationDelta(10.0)
    s.analyzePattern(A)
    s.factorize(A)
    o = OracleSymLDLT(s.symbolicFactor())
    o.setExpectedSignPattern(sign)
    o.set(mode=1, initial_delta=10.0)
    o.factorize(A)
    assert s.inertia().as_tuple() == o.inertia()
    assert s.numPerturbedPivots() == o.info()["num_perturbed"] >= weak
    assert abs(s.totalPerturbation() - o.info()["total_perturbation"]) <= 1e-9 * max(1.0, s.totalPerturbation())
    if weak == 0:
        X = st = Stream(n).normal(2 * n).reshape(2, n).T
        B = np.asfortranarray(K @ X)
        R = K @ s.solve(B) - B
        bw = np.abs(R).max() / (np.abs(K).sum(axis=1).max() * np.abs(X).max() + np.abs(B).max())
        assert bw < 100 * n * 2.0 ** -53  # backward stable on a quasi-definite matrix


@pytest.mark.gpu
def test_static_fronts_of_different_heights():
    """Short and tall dense fronts in one level: the launches cover the tallest,
    so most CTAs of a short front's column have no rows, and the short ones are
    finished panels earlier. Every front as the oracle has it, and the same bits
    at every repetition."""
    sizes = [129, 801, 140, 545, 289, 1025, 130]
    blocks = [quasi_definite(n, n // 3, 2) for n in sizes]
    K, sign = sp.csc_matrix(sp.block_diag([sp.coo_array(b) for b, _ in blocks])), np.concatenate([g for _, g in blocks])
    A = lower(K)
    s = SymLDLT()
    s.setMode(Mode.StaticRegularized)
    s.setOrdering(OrderingType.Natural)
    s.setExpectedSignPattern(sign)
    s.setInitialRegularizationDelta(10.0)
    s.analyzePattern(A)
    s.factorize(A)
    o = OracleSymLDLT(s.symbolicFactor())
    o.setExpectedSignPattern(sign)
    o.set(mode=1, initial_delta=10.0)
    o.factorize(A)
    assert s.inertia().as_tuple() == o.inertia()
    assert s.numPerturbedPivots() == o.info()["num_perturbed"] >= 2 * len(sizes)
    d0 = [f.Ddiag.copy() for f in s.numericFactor().fronts]
    for fs, fo in zip(s.numericFactor().fronts, o.fronts()):
        assert fs.nPivots == fo["nPivots"] and list(fs.rowIndices) == list(fo["rowIndices"])
        np.testing.assert_allclose(fs.Ddiag, fo["Ddiag"], rtol=1e-9, atol=1e-9)
    for _ in range(3):
        s.refactorize(A)
        for f, d in zip(s.numericFactor().fronts, d0):
            np.testing.assert_array_equal(f.Ddiag, d)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [129, 255, 256, 257, 512, 513, 784, 785, 1025, 1057, 1288])
def test_threshold_dense_front(n):
    """Fronts whose pivots need interchanges and 2x2 blocks, at the edges of
    the single-CTA panel's two widths and of its range, and in the cluster
    panel (runs that stop inside a panel and start again): inertia from the
    eigenvalues, backward error of a solve."""
    st = Stream(n)
    G = st.normal(n * n).reshape(n, n)
    K = (G + G.T) / 2
    K[np.arange(0, n, 3), np.arange(0, n, 3)] += 3 * np.sqrt(n)
    s = SymLDLT()
    s.setOrdering(OrderingType.Natural)
    A = lower(sp.csc_matrix(K))
    s.analyzePattern(A)
    s.factorize(A)
    w = np.linalg.eigvalsh(K)
    assert np.abs(w).min() > 1e-9 * np.abs(w).max()
    assert s.inertia().as_tuple() == (int((w > 0).sum()), int((w < 0).sum()), 0)
    x = Stream(n + 1).normal(n)
    b = K @ x
    r = K @ s.solve(b) - b
    # Bunch-Kaufman growth on a random matrix is far below the 1e3 allowed here
    assert np.abs(r).max() < 1e3 * n * 2.0 ** -53 * np.abs(K).sum(axis=1).max() * np.abs(x).max()


def set_cluster(s, ctas):
    """The panel's cluster size on every level (1: the single-CTA kernels)."""
    lib = L.load()
    for lv in range(int(s.plan_stats()["levels"])):
        assert lib.symla_gpu_set_level_schedule(s._ctx.h, lv, 0, ctas) == L.SYMLA_OK


@pytest.mark.gpu
@pytest.mark.parametrize("ctas", [2, 4, 8, 16])
def test_restart_after_interchange(ctas):
    """Panels of one cluster that interchange rows of the front and then
    speculate again on the rows just moved (read back from the front by bulk
    copies): the pivots, kinds and factor of the CPU oracle, and the same bits
    at every repetition."""
    n = 600
    st = Stream(n)
    G = st.normal(n * n).reshape(n, n)
    K = (G + G.T) / 2
    # plain pivots with a zero diagonal now and then: a 2x2 or an interchange
    # with a far row, then plain pivots again in the same panel
    K[np.arange(n), np.arange(n)] += np.where(np.arange(n) % 2 == 0, 3.0, -3.0) * n
    K[5::23, 5::23] = 0.0
    A = lower(sp.csc_matrix(K))
    s = SymLDLT()
    s.setOrdering(OrderingType.Natural)
    s.analyzePattern(A)
    s.factorize(A)
    set_cluster(s, ctas)
    s.refactorize(A)
    stats = s.plan_stats()
    assert stats["seq_interchange"] + stats["seq_2x2"] >= 10
    o = OracleSymLDLT(s.symbolicFactor())
    o.factorize(A)
    assert s.inertia().as_tuple() == o.inertia()
    fs, fo = s.numericFactor().fronts[0], o.fronts()[0]
    assert list(fs.rowIndices) == list(fo["rowIndices"])
    assert [(b.start, b.kind) for b in fs.pivotBlocks] == fo["pivotBlocks"]
    np.testing.assert_allclose(np.tril(fs.L, -1), np.tril(fo["L"], -1), rtol=0, atol=1e-10 * np.abs(fo["L"]).max())
    for _ in range(3):
        s.refactorize(A)
        np.testing.assert_array_equal(s.numericFactor().fronts[0].L, fs.L)


@pytest.mark.gpu
@pytest.mark.parametrize("last", [1, 2, 7, 8, 9, 15, 16, 17, 24, 25, 31, 32])
def test_diagonal_block_sizes(last):
    """A diagonal block of every kind of size (one warp, steps of eight
    columns): D against the oracle, and the same bits at every repetition."""
    n = 128 + last
    K, sign = quasi_definite(n, n // 3, 2)
    A = lower(sp.csc_matrix(K))
    s = SymLDLT()
    s.setMode(Mode.StaticRegularized)
    s.setOrdering(OrderingType.Natural)
    s.setExpectedSignPattern(sign)
    s.setInitialRegularizationDelta(10.0)
    s.analyzePattern(A)
    s.factorize(A)
    o = OracleSymLDLT(s.symbolicFactor())
    o.setExpectedSignPattern(sign)
    o.set(mode=1, initial_delta=10.0)
    o.factorize(A)
    f = s.numericFactor().fronts[0]
    # quasi-definite, no growth: n eps times the condition of the leading blocks
    np.testing.assert_allclose(f.Ddiag, o.fronts()[0]["Ddiag"], rtol=1e-10, atol=1e-10)
    for _ in range(10):
        s.refactorize(A)
        np.testing.assert_array_equal(s.numericFactor().fronts[0].L, f.L)


@pytest.mark.gpu
def test_restart_sums_earlier_pivots_apart():
    """A speculation that restarts late in a panel takes the 26 earlier pivots'
    products from entries a thousand times their size. Summed apart, an entry of
    [1, 2) is rounded twice (the two subtractions) and its quotient once, 0.29
    ulp each in the root mean square, about 0.6 with the quotient's slack;
    subtracted one by one it would be rounded 26 times, 1.5 ulp. The values
    before scaling against 80-bit arithmetic."""
    n, p0, d0 = 400, 26, 1024.0
    st = Stream(n)
    U = st.uniform(n * n, 1.0, 2.0) * np.where(st.uniform(n * n) < 0.5, -1.0, 1.0)
    K = np.tril(U.reshape(n, n), -1)
    K = K + K.T
    K[np.arange(n), np.arange(n)] = d0 * np.where(np.arange(n) % 3 == 0, -1.0, 1.0)
    K[p0 - 2, p0 - 2] = 0.0  # an interchange, then one plain pivot decided alone, then the restart
    A = lower(sp.csc_matrix(K))
    s = SymLDLT()
    s.setOrdering(OrderingType.Natural)
    s.analyzePattern(A)
    s.factorize(A)
    set_cluster(s, 2)
    s.refactorize(A)
    f = s.numericFactor().fronts[0]
    rows = np.asarray(f.rowIndices)
    assert rows[p0 - 2] != p0 - 2 and all(b.kind == 0 for b in f.pivotBlocks[:32])
    P = K[np.ix_(rows, rows)].astype(np.longdouble)[:, :32]
    for k in range(32):
        for j in range(k):
            P[k:, k] -= P[k:, j] * (P[k, j] / P[j, j])
    V = f.L[32:, :32] * f.Ddiag[:32]
    err = (V - P[32:]).astype(np.float64) / 2.0 ** -52
    rms = np.sqrt((err ** 2).mean(axis=0))
    assert rms[p0:].max() < 1.0, rms[p0:]


@pytest.mark.gpu
@pytest.mark.parametrize("n", [160, 285, 600, 784, 785, 1100])
@pytest.mark.parametrize("ctas", [1, 2, 4])
def test_panel_kernels_take_the_oracles_pivots(n, ctas):
    """The single-CTA panels (with L in shared memory up to 784 rows, reading it
    back above) and clusters on the same fronts, several outer blocks of 256
    pivots with interchanges and 2x2 pivots throughout: the oracle's pivot
    order, kinds and factor."""
    G = Stream(n).normal(n * n).reshape(n, n)
    K = (G + G.T) / 2
    K[np.arange(0, n, 3), np.arange(0, n, 3)] += 3 * np.sqrt(n)
    A = lower(sp.csc_matrix(K))
    s = SymLDLT()
    s.setOrdering(OrderingType.Natural)
    s.analyzePattern(A)
    s.factorize(A)
    set_cluster(s, ctas)
    s.refactorize(A)
    o = OracleSymLDLT(s.symbolicFactor())
    o.factorize(A)
    fs, fo = s.numericFactor().fronts[0], o.fronts()[0]
    assert s.inertia().as_tuple() == o.inertia()
    assert list(fs.rowIndices) == list(fo["rowIndices"])
    assert [(b.start, b.kind) for b in fs.pivotBlocks] == fo["pivotBlocks"]
    assert sum(b.kind for b in fs.pivotBlocks) > n // 20 and list(fs.rowIndices) != sorted(fs.rowIndices)
    # growth times the rounding of n sums
    scale = np.abs(fo["L"]).max() * n * 2.0 ** -53 * 1e4
    np.testing.assert_allclose(np.tril(fs.L, -2), np.tril(fo["L"], -2), rtol=0, atol=scale)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [129, 256, 300, 784, 785, 900])
def test_static_single_cta(n):
    """The static branches of the single-CTA panels, against the oracle."""
    K, sign = quasi_definite(n, n // 3, 3)
    A = lower(sp.csc_matrix(K))
    s = SymLDLT()
    s.setMode(Mode.StaticRegularized)
    s.setOrdering(OrderingType.Natural)
    s.setExpectedSignPattern(sign)
    s.setInitialRegularizationDelta(10.0)
    s.analyzePattern(A)
    s.factorize(A)
    set_cluster(s, 1)
    s.refactorize(A)
    o = OracleSymLDLT(s.symbolicFactor())
    o.setExpectedSignPattern(sign)
    o.set(mode=1, initial_delta=10.0)
    o.factorize(A)
    assert s.inertia().as_tuple() == o.inertia()
    assert s.numPerturbedPivots() == o.info()["num_perturbed"] >= 3
    fs, fo = s.numericFactor().fronts[0], o.fronts()[0]
    np.testing.assert_allclose(fs.Ddiag, fo["Ddiag"], rtol=1e-10, atol=1e-10)
    np.testing.assert_allclose(np.tril(fs.L, -1), np.tril(fo["L"], -1), rtol=0, atol=1e-10)
