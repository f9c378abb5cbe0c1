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


@pytest.mark.gpu
def test_memory_of_replanned_fronts_follows_their_use():
    """Factorizations that delay one pivot more each time: what the context
    holds beyond its plan stays near what the largest of them needs (a dense
    front of about 1540 rows), and goes back when nothing is delayed any more."""
    import torch
    m, leaves = 1500, 40
    base = leaves_on_a_dense_root(m, leaves, 0)
    lead = [base.indptr[i] for i in range(leaves)]  # the leaves' diagonal entries
    assert all(base.indices[p] == i and base.data[p] == 3.0 for i, p in enumerate(lead))
    s = SymLDLT()
    s.setOrdering(OrderingType.Natural)
    s.analyzePattern(base, SymbolicFactorOptions(0, 0.0))

    def held(zeros):
        A = base.copy()
        for i, p in enumerate(lead):
            A.data[p] = 0.0 if i < zeros else 3.0
        s.factorize(A)
        assert s.last_info.num_delayed == zeros
        torch.cuda.synchronize()
        return -torch.cuda.mem_get_info()[0]

    plan = held(0)
    front = 8 * (m + leaves) ** 2
    used = [held(z) - plan for z in range(2, leaves, 3)]
    # an eighth ahead, the packed operands of the enlarged front (17 chunks of 16
    # pivots), the driver's 2 MB pages of the few arrays beside them
    packed = 2 * 17 * ((m + leaves) // 64 + 1) * 16 * 68 * 8
    assert max(used) < 1.25 * front + packed + 6 * 2 ** 20, (used, front, packed)
    held(0)
    assert held(0) - plan < 0.25 * front
