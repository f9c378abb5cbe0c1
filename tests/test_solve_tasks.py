"""The solves' task shapes, against dense solutions: fronts of at most 32 rows
(a warp each) and one more, block and pivot counts that are odd or a multiple
of 64, 2x2 pivots on block boundaries, and right-hand-side counts at the edges
of a half, a whole and several groups of 16."""
import numpy as np
import pytest
import scipy.sparse as sp

from ma57_b200 import OrderingType, SymLDLT
from ma57_b200 import matrices as M
from ma57_b200.solver import SymbolicFactorOptions


def check(A, nrhs, ordering):
    s = SymLDLT()
    s.setOrdering(ordering)
    s.analyzePattern(A, SymbolicFactorOptions())
    s.factorize(A)
    F = M.sym_full(A).toarray()
    n = A.shape[0]
    B = M.Stream(n + nrhs).normal(n * nrhs).reshape(nrhs, n).T
    X = s.solve(np.asfortranarray(B))
    R = F @ X - B
    # column-wise backward error, growth of the factorization included
    err = np.abs(R).max(axis=0) / (np.abs(F).sum(axis=1).max() * np.abs(X).max(axis=0))
    assert err.max() < 100 * n * 2.0 ** -53
    X1 = s.solve(np.asfortranarray(B))
    np.testing.assert_array_equal(X, X1)
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("nrhs", [1, 7, 8, 9, 16, 17, 33, 64, 65, 130])
def test_right_hand_side_groups(nrhs):
    A, _ = M.config1(9)
    check(A, nrhs, OrderingType.AMD)


def two_block(n1, n2, pairs, seed):
    """Two dense leaves of n1 and a dense separator of n2 columns; with
    `pairs`, a zero diagonal in the leaves' and separator's first columns so
    that 2x2 pivots appear throughout."""
    st = M.Stream(seed)
    n = 2 * n1 + n2
    G = st.normal(n * n).reshape(n, n)
    K = (G + G.T) / 2
    K[:n1, n1:2 * n1] = 0.0
    K[n1:2 * n1, :n1] = 0.0
    d = np.arange(n)
    K[d, d] = 0.0 if pairs else np.where(d % 2 == 0, 1.0, -1.0) * 2 * np.sqrt(n)
    return M.lower(sp.csc_matrix(K))


@pytest.mark.gpu
@pytest.mark.parametrize("n1,n2", [(3, 29), (5, 28), (16, 16), (20, 13), (63, 64), (65, 63), (64, 129), (129, 65), (191, 67)])
@pytest.mark.parametrize("pairs", [False, True])
@pytest.mark.parametrize("nrhs", [1, 12])
def test_block_edges(n1, n2, pairs, nrhs):
    check(two_block(n1, n2, pairs, 31 * n1 + n2), nrhs, OrderingType.Natural)
