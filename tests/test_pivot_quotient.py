"""The panels' division by a pivot (a Newton reciprocal and a residual step,
ma57_b200/csrc/gpu/panel_block.cuh) against the correctly rounded division:
tests/cpp/pivot_quotient_test.cu."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest
import scipy.sparse as sp

from ma57_b200 import OrderingType, SymLDLT
from ma57_b200 import _lib as L
from ma57_b200 import build as B
from ma57_b200 import matrices as M
from ma57_b200.solver import as_csc

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "cpp", "pivot_quotient_test.cu")
OUT = os.path.join(ROOT, "tests", "cpp", "_build", "pivot_quotient_test")


def compile_test():
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    cmd = [B.NVCC, *B.ARCH, "-std=c++17", "-O3", "--expt-relaxed-constexpr", "-I",
           os.path.join(ROOT, "ma57_b200", "csrc", "gpu"), SRC, "-o", OUT]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


def test_compiles():
    compile_test()


@pytest.mark.gpu
def test_quotients_match_the_division():
    compile_test()
    r = subprocess.run([OUT], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [L.MODE_THRESHOLD, L.MODE_STATIC])
@pytest.mark.parametrize("c", [0, 45])
@pytest.mark.parametrize("n,ctas", [(20, 0), (100, 0), (300, 2), (300, 1), (800, 1), (800, 16)])
def test_pivots_whose_reciprocal_overflows(n, ctas, c, mode):
    """A column whose pivot is 2^-1030 over entries of a sixteenth of whole
    multiples of it, in every kernel's range: its L is that of the numbers
    scaled back (to the 2^-40 that subnormal numbers of that size keep), not
    NaN."""
    c = min(c, n - 2)
    st = M.Stream(n)
    G = st.normal(n * n).reshape(n, n)
    K = (G + G.T) / 2 + 4 * n * np.eye(n)
    k = st.integers(n, 15) + 1.0
    want = (k[c + 1:] - K[c + 1:, :c] @ np.linalg.solve(K[:c, :c], k[:c])) / 16
    K[c, :] = K[:, c] = k * 2.0 ** -1034
    K[c, c] = 2.0 ** -1030
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
    o.mode = mode
    o.zero_tolerance = o.relative_pivot_floor = o.static_rel_floor = o.static_abs_floor = 0.0
    o.static_delta = 1.0
    assert lib.symla_gpu_factorize(h, L.ptr_d(vals), 0, C.byref(o), C.byref(info)) == L.SYMLA_OK
    s._after_factor(s._ctx, info)
    assert info.num_perturbed == 0 and info.n_pos == n
    f = s.numericFactor().fronts[0]
    assert list(f.rowIndices) == list(range(n)) and np.isfinite(f.L).all()
    np.testing.assert_allclose(f.L[c + 1:, c], want, rtol=0, atol=1e-9)
