"""Assembly of large fronts with many children, against the CPU oracle: more
children than one staging batch of the assembly holds in every 32-column
block, at the edges of its column blocks and row chunks, with and without
delayed pivots (the re-planned front's child lists)."""
import numpy as np
import pytest
import scipy.sparse as sp

from ma57_b200 import OrderingType, SymLDLT
from ma57_b200.matrices import Stream, lower, sym_full
from ma57_b200.solver import SymbolicFactorOptions
from oracle.pyoracle import OracleSymLDLT


def leaves_on_a_dense_root(m, leaves, zero_leaves):
    """`leaves` single columns, each coupled to three rows of a dense m x m
    block ordered last; the first `zero_leaves` have a zero diagonal, so
    their pivots are delayed to the dense front."""
    st = Stream(7 * m + leaves)
    n = leaves + m
    D = st.normal(m * m).reshape(m, m)
    A = np.zeros((n, n))
    A[leaves:, leaves:] = (D + D.T) / 2 + 4 * np.sqrt(m) * np.diag(np.where(np.arange(m) % 3 == 0, -1.0, 1.0))
    for i in range(leaves):
        A[i, i] = 0.0 if i < zero_leaves else 3.0
        r = leaves + np.unique(st.integers(3, m))
        A[r, i] = A[i, r] = st.uniform(len(r), 0.5, 1.5)
    S = sp.tril(sp.csc_matrix(A)).tolil()
    for i in range(zero_leaves):
        S[i, i] = 0.0
    return lower(sp.csc_matrix(S))


@pytest.mark.gpu
@pytest.mark.parametrize("m", [129, 160, 513, 545])
@pytest.mark.parametrize("leaves,zero_leaves", [(150, 0), (150, 5), (600, 0)])
def test_many_children(m, leaves, zero_leaves):
    A = leaves_on_a_dense_root(m, leaves, zero_leaves)
    s = SymLDLT()
    s.setOrdering(OrderingType.Natural)
    s.analyzePattern(A, SymbolicFactorOptions(0, 0.0))
    s.factorize(A)
    o = OracleSymLDLT(s.symbolicFactor())
    o.factorize(A)
    assert s.inertia().as_tuple() == o.inertia()
    assert s.last_info.num_delayed == zero_leaves
    F = sym_full(A)
    X = Stream(m).normal(2 * A.shape[0]).reshape(2, -1).T
    B = np.asfortranarray(F @ X)
    R = F @ s.solve(B) - B
    # backward stable: a modest multiple of n eps, pivot growth included
    bw = np.abs(R).max() / (abs(F).sum(axis=1).max() * np.abs(X).max() + np.abs(B).max())
    assert bw < 100 * A.shape[0] * 2.0 ** -53
