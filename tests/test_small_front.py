"""Small fronts (one dense front, natural order) at the edges of the warp's
32 rows, the 16-pivot panels and the kernel's 128 rows, against the CPU
oracle: the same pivot order and kinds, inertia and factor."""
import numpy as np
import pytest
import scipy.sparse as sp

from ma57_b200 import Mode, OrderingType, SymLDLT, autotune
from ma57_b200 import matrices as M
from ma57_b200.solver import SymbolicFactorOptions
from oracle.pyoracle import OracleSymLDLT

SIZES = [2, 31, 32, 33, 34, 48, 49, 64, 65, 97, 113, 127, 128]


def dense(n, kind):
    G = M.Stream(17 * n + len(kind)).normal(n * n).reshape(n, n)
    K = (G + G.T) / 2
    d = np.arange(n)
    if kind == "plain":
        K[d, d] += np.where(d % 2 == 0, 1.0, -1.0) * 3 * n
    elif kind == "pairs":
        K[d, d] = 0.0
    return K


def compare(s, o, scale):
    assert s.inertia().as_tuple() == o.inertia()
    for fs, fo in zip(s.numericFactor().fronts, o.fronts()):
        assert list(fs.rowIndices) == list(fo["rowIndices"])
        assert [(b.start, b.kind) for b in fs.pivotBlocks] == fo["pivotBlocks"]
        # L is determined up to rounding: growth times n eps
        np.testing.assert_allclose(np.tril(fs.L, -1), np.tril(fo["L"], -1), rtol=0, atol=scale)
        np.testing.assert_allclose(fs.Ddiag, fo["Ddiag"], rtol=scale, atol=scale)


@pytest.mark.gpu
@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("kind", ["plain", "pairs", "random"])
def test_threshold(n, kind):
    A = M.lower(sp.csc_matrix(dense(n, kind)))
    s = SymLDLT()
    s.setOrdering(OrderingType.Natural)
    s.analyzePattern(A)
    s.factorize(A)
    o = OracleSymLDLT(s.symbolicFactor())
    o.factorize(A)
    compare(s, o, 1e-9)


@pytest.mark.gpu
@pytest.mark.parametrize("n", SIZES)
def test_static(n):
    K = dense(n, "plain")
    sign = np.where(np.arange(n) % 2 == 0, 1, -1)
    # the first pivot has no Schur complement: its wrong sign is certain
    K[0, 0] = -1e-3 * sign[0]
    A = M.lower(sp.csc_matrix(K))
    s = SymLDLT()
    s.setMode(Mode.StaticRegularized)
    s.setOrdering(OrderingType.Natural)
    s.setExpectedSignPattern(sign)
    s.setInitialRegularizationDelta(3.0 * n)
    s.analyzePattern(A)
    s.factorize(A)
    o = OracleSymLDLT(s.symbolicFactor())
    o.setExpectedSignPattern(sign)
    o.set(mode=1, initial_delta=3.0 * n)
    o.factorize(A)
    assert s.numPerturbedPivots() == o.info()["num_perturbed"] >= 1
    compare(s, o, 1e-9)


@pytest.mark.gpu
@pytest.mark.parametrize("m", [33, 64, 100])
@pytest.mark.parametrize("leaves,zero_leaves", [(40, 0), (40, 4), (90, 0)])
def test_children(m, leaves, zero_leaves):
    """More children than one staging batch, and delayed ones, under a small front."""
    from test_assembly_many_children import leaves_on_a_dense_root
    A = leaves_on_a_dense_root(m, leaves, zero_leaves)
    s = SymLDLT()
    s.setOrdering(OrderingType.Natural)
    s.analyzePattern(A, SymbolicFactorOptions(0, 0.0))
    s.factorize(A)
    o = OracleSymLDLT(s.symbolicFactor())
    o.factorize(A)
    assert s.last_info.num_delayed == zero_leaves
    compare(s, o, 1e-9)


def factor_both(A, ordering, options=None):
    s = SymLDLT()
    s.setOrdering(ordering)
    s.analyzePattern(A, options or SymbolicFactorOptions())
    s.factorize(A)
    o = OracleSymLDLT(s.symbolicFactor())
    o.factorize(A)
    return s, o


@pytest.mark.gpu
@pytest.mark.parametrize("every", [0, 15])
def test_warp_per_front(every):
    """Levels whose small fronts all have at most 32 rows: a warp each, with
    children, 2x2 pivots and interchanges; a zero on every 15th diagonal delays
    pivots too. (Random values: no ties for rounding to decide.)"""
    blocks = []
    for i in (0, 2, 3, 6):  # (regular with the zeros too)
        n = 120 + 10 * i
        S = M.random_sparse_spd(n, 4, 50 + i) - sp.identity(n) * 2.0
        S = sp.coo_matrix(sp.tril(S))
        if every:
            S.data[(S.row == S.col) & (S.row % every == 0)] = 0.0
        blocks.append(sp.coo_array(S))
    A = sp.csc_matrix(sp.block_diag(blocks))
    s, o = factor_both(A, OrderingType.AMD)
    assert any(i["small"] and i["small_max_m"] <= 32 for i in autotune.level_info(s))
    assert (s.last_info.num_delayed > 0) == (every > 0)
    assert any(b.kind for f in s.numericFactor().fronts for b in f.pivotBlocks)
    compare(s, o, 1e-9 * max(np.abs(f["L"]).max() for f in o.fronts() if f["L"].size))


@pytest.mark.gpu
@pytest.mark.parametrize("leaves", [1000, 1535, 1536, 1700])
def test_level_of_warp_and_cta_fronts(leaves):
    """On either side of the number of warp-sized fronts (1536) from which those
    of a level take a launch of their own beside the larger ones; four of them
    delay their pivot to a front that is assembled from all of them."""
    from test_assembly_many_children import leaves_on_a_dense_root
    tree = leaves_on_a_dense_root(100, leaves, 4)
    blocks = [tree] + [M.lower(sp.csc_matrix(dense(n, "random"))) for n in (33, 40, 64, 127, 128)]
    A = sp.csc_matrix(sp.block_diag([sp.coo_array(b) for b in blocks]))
    s, o = factor_both(A, OrderingType.Natural, SymbolicFactorOptions(0, 0.0))
    info = autotune.level_info(s)[0]
    assert info["small"] == leaves + 5 and info["small_max_m"] == 128
    assert s.last_info.num_delayed == 4
    compare(s, o, 1e-9)
