"""The work this solver is measured on: factorizations, refactorizations and
solves as a user's program issues them, over the sizes of the benchmark
configurations and tests, from one 210-unknown system to the 64^3 stencil.

A pass goes through the Python mirror of SymLDLT (host arrays in and out) or
through the C ABI with arrays that stay on the device, as include/symla_gpu.h
documents. Every matrix has its pattern from the case and its values from the
seed; the symbolic analysis, the device context and (for the solve cases) the
factorization are what such a program keeps.

Matrix values are multiples of 2^-20 (2^-27 and 2^-33 in the KKT
regularisation blocks) and solutions multiples of 2^-10, and the right-hand
sides are formed from the solutions, so every product and sum of B = A X is
exact in 64 bits: the drawn X is the exact solution of the system, at any
size.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from ma57_b200 import _lib as L
from ma57_b200 import matrices as M
from ma57_b200.batch import BatchedSolver
from ma57_b200.solver import (Analysis, Context, GmresRefinementOptions, Mode, OrderingType, RefinementOptions,
                              SymbolicFactorOptions, SymLDLT, as_csc)

# --------------------------------------------------------------------------
# Cases


def listed():
    return [
        # one small 2D system of the many-systems configuration, served alone:
        # latency of a refactorization and a solve through the Python API
        dict(name="grid2_210", kind="grid2", a=14, b=15, nrhs=1),
        # the top of that configuration's range, its 8 right-hand sides
        dict(name="grid2_3922", kind="grid2", a=53, b=74, nrhs=8),
        # the many-systems configuration served in batches: 256 systems as
        # one block-diagonal factorization
        dict(name="batch_256", kind="batch", count=256, nrhs=8),
        # the first configuration: indefinite 7-point Laplacian, AMD, values
        # and right-hand side on the device, ordinary launches
        dict(name="grid3_20", kind="grid3", k=20, stencil=7, ordering="amd", nrhs=1, precision="fp64", graph=False),
        # a ragged mid-size 27-point grid, nested dissection, graph launch,
        # an odd number of right-hand sides
        dict(name="grid3_27", kind="grid3", k=27, stencil=27, ordering="metis", nrhs=3, precision="fp64", graph=True),
        # the mixed-precision option with its refinement
        dict(name="grid3_32_mixed", kind="grid3", k=32, stencil=27, ordering="metis", nrhs=16, precision="mixed",
             graph=True),
        # the benchmark's step: 64^3 27-point stencil, 16 right-hand sides
        dict(name="grid3_64", kind="grid3", k=64, stencil=27, ordering="metis", nrhs=16, precision="fp64", graph=True),
        # solves with a factorization that is kept: one right-hand side (a
        # time step, a Krylov preconditioner) and many (a block of loads)
        dict(name="solve_40_1", kind="solve", k=40, nrhs=1),
        dict(name="solve_48_37", kind="solve", k=48, nrhs=37),
        # the second configuration: KKT with StaticRegularized and refinement
        dict(name="kkt_200", kind="kkt", grid=200, n2=20000, nrhs=1),
        # one step of the interior-point sequence: static pivoting, GMRES-IR
        dict(name="ipm_16", kind="ipm", k=16, nrhs=1),
        # a grid with tie constraints (multipliers with a zero block) under
        # threshold pivoting: the multipliers' pivots are delayed to the
        # parents (the re-planned path)
        dict(name="ties_40", kind="ties", grid=40, n2=311, nrhs=2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["grid2", "batch", "grid3", "grid3", "solve", "kkt", "ipm", "ties"])
    if kind == "grid2":
        n, r = _log(rng, 200, 4000), math.exp(rng.uniform(math.log(0.25), math.log(4.0)))
        a = max(2, int(round(math.sqrt(n * r))))
        return dict(kind=kind, a=a, b=max(2, n // a), nrhs=_log(rng, 1, 16))
    if kind == "batch":
        return dict(kind=kind, count=_log(rng, 16, 256), nrhs=_log(rng, 1, 16))
    if kind == "grid3":
        stencil = rng.choice([7, 27])
        return dict(kind=kind, k=_log(rng, 9, 48), stencil=stencil,
                    ordering="amd" if stencil == 7 and rng.random() < 0.5 else "metis", nrhs=_log(rng, 1, 40),
                    precision="mixed" if rng.random() < 0.25 else "fp64", graph=rng.random() < 0.6)
    if kind == "solve":
        return dict(kind=kind, k=_log(rng, 9, 48), nrhs=_log(rng, 1, 64))
    if kind == "kkt":
        g = _log(rng, 20, 150)
        return dict(kind=kind, grid=g, n2=int(g * g * rng.uniform(0.2, 0.5)), nrhs=_log(rng, 1, 8))
    if kind == "ipm":
        return dict(kind=kind, k=_log(rng, 8, 20), nrhs=_log(rng, 1, 4))
    g = _log(rng, 12, 100)
    return dict(kind=kind, grid=g, n2=max(2, int(g * g * rng.uniform(0.02, 0.3))), nrhs=_log(rng, 1, 8))


# --------------------------------------------------------------------------
# Matrices: the pattern from the case, the values from the seed


def _quant(v, bits):
    return np.round(v * 2.0 ** bits) / 2.0 ** bits


def _stencil(case):
    if case["kind"] == "grid2":
        return M.lower(M.laplacian5(case["a"], case["b"])), 2.0
    if case.get("stencil", 27) == 7:
        return M.lower(M.laplacian7(case["k"])), 2.0
    return M.lower(M.laplacian27(case["k"])), 3.0


def _vary(A, shift, rng):
    """Couplings within 5 % of the stencil's, the diagonal minus the shift."""
    A = A.copy()
    col = np.repeat(np.arange(A.shape[0]), np.diff(A.indptr))
    w = rng.uniform(-0.05, 0.05, A.nnz)
    A.data = _quant(np.where(col == A.indices, A.data - shift + 2 * w, A.data * (1 + w)), 20)
    return A


@functools.lru_cache(maxsize=4)
def _coupling(n1, n2):
    return M.random_coupling(n2, n1, 3, M.Stream(M.SEED_BASE + 2))


@functools.lru_cache(maxsize=4)
def _ties(n1, n2):
    """n2 constraints x_i - x_j = b, each on two vertical neighbours of the
    square grid, no node in two of them."""
    g = math.isqrt(n1)
    p = np.sort(np.random.default_rng([g, n2]).permutation((g // 2) * g)[:n2])
    i = (p // g) * 2 * g + p % g
    cols, rows = np.concatenate([i, i + g]), np.tile(np.arange(n2), 2)
    return M.sp.csc_matrix((np.repeat([1.0, -1.0], n2), (rows, cols)), shape=(n2, n1))


def _matrix(case, seed):
    """Lower triangle of the case's matrix, and (n1, n2) of a KKT system."""
    rng = np.random.default_rng([seed, 1])
    if case["kind"] in ("grid2", "grid3", "solve"):
        A, shift = _stencil(case)
        return _vary(A, shift, rng), None
    if case["kind"] == "ipm":
        n1 = case["k"] ** 3
        n2 = n1 // 2
        E = M.laplacian7(case["k"])
        # the barrier diagonal of a step in the middle of the sequence
        E.setdiag(E.diagonal() + _quant(1e-4 * np.exp(-2.0 * rng.uniform(math.log(1e-3), math.log(1e2), n1)), 20))
        f = 2.0 ** -33
    else:
        n1, n2 = case["grid"] ** 2, case["n2"]
        E = M.laplacian5(case["grid"], case["grid"])
        E.setdiag(E.diagonal() + _quant(1e-2 + 1e-2 * rng.random(n1), 20))
        f = 2.0 ** -27
    A = (_ties if case["kind"] == "ties" else _coupling)(n1, n2).copy()
    A.data = _quant(A.data + 0.1 * rng.standard_normal(A.nnz), 20)
    F = E[:n2, :n2] * 0.0
    if case["kind"] != "ties":
        F.setdiag(f)
    F.eliminate_zeros()
    return M.kkt(E, F, A), (n1, n2)


def _solution(n, nrhs, seed, part=0):
    rng = np.random.default_rng([seed, 2, part])
    return _quant(rng.standard_normal((nrhs, n)), 10).T  # column-major n x nrhs


def _rhs(A, X):
    return np.asfortranarray(M.sym_full(A) @ X)


def _systems(case, seed):
    """The batch's systems: rectangles with n log-uniform in [200, 4000]."""
    out = []
    for i in range(case["count"]):
        S, _, _, _ = M.config4_system(i)
        S = _vary(S, 0.0, np.random.default_rng([seed, 3, i]))
        out.append((S, _solution(S.shape[0], case["nrhs"], seed, i)))
    return out


@functools.lru_cache(maxsize=4)
def _analysis(key):
    """The symbolic analysis of a pattern, shared by every matrix on it."""
    case = dict(key)
    A, _ = _matrix(case, 0)
    n, cp, ri, _ = as_csc(A)
    o = {"amd": OrderingType.AMD, "metis": OrderingType.Metis}[case["ordering"]]
    return Analysis(n, cp, ri, o, SymbolicFactorOptions())


def _pattern_key(case):
    if case["kind"] in ("grid3", "solve"):
        return (("kind", "grid3"), ("k", case["k"]), ("stencil", case.get("stencil", 27)),
                ("ordering", case.get("ordering", "metis")))
    if case["kind"] == "grid2":
        return (("kind", "grid2"), ("a", case["a"]), ("b", case["b"]), ("ordering", "amd"))
    if case["kind"] == "ipm":
        return (("kind", "ipm"), ("k", case["k"]), ("ordering", "amd"))
    return (("kind", case["kind"]), ("grid", case["grid"]), ("n2", case["n2"]), ("ordering", "amd"))


# --------------------------------------------------------------------------
# What a program holds, and one pass


def _check(rc):
    if rc != L.SYMLA_OK:
        raise RuntimeError(L.last_error())


def _dev(t):
    return C.cast(C.c_void_p(t.data_ptr()), C.POINTER(C.c_double))


class DeviceSystem:
    """A program on the C ABI whose arrays live on the device."""

    def __init__(self, case, seed):
        A, _ = _matrix(case, seed)
        n, cp, ri, vals = as_csc(A)
        X = _solution(n, case["nrhs"], seed)
        self.case, self.n = case, n
        self.ctx = Context(_analysis(_pattern_key(case)), cp, ri, torch.cuda.current_device())
        self.values = torch.from_numpy(vals).cuda()
        self.B = torch.from_numpy(np.ascontiguousarray(_rhs(A, X).T)).cuda()  # row r: right-hand side r
        self.opts = L.FactorOpts()
        L.load().symla_factor_opts_default(C.byref(self.opts))
        if case.get("precision") == "mixed":
            self.opts.precision = L.PREC_MIXED
        L.load().symla_gpu_set_graph(self.ctx.h, int(case.get("graph", True)))
        torch.cuda.synchronize()
        if case["kind"] == "solve":
            self.factorize()

    def factorize(self):
        info = L.FactorInfo()
        _check(L.load().symla_gpu_factorize(self.ctx.h, _dev(self.values), 1, C.byref(self.opts), C.byref(info)))
        return torch.tensor([info.n_pos, info.n_neg, info.n_zero])

    def solve(self):
        X = torch.empty_like(self.B)
        _check(L.load().symla_gpu_solve(self.ctx.h, _dev(self.B), self.n, self.case["nrhs"], _dev(X), self.n, 1))
        return X

    def solve_refined(self):
        X, ri = torch.empty_like(self.B), L.RefineInfo()
        _check(L.load().symla_gpu_solve_refine(self.ctx.h, _dev(self.values), _dev(self.B), self.n,
                                               self.case["nrhs"], _dev(X), self.n, 1, 10, 1e-12, C.byref(ri)))
        return X


class HostSystem:
    """A program on the Python mirror of SymLDLT, with host arrays."""

    def __init__(self, case, seed):
        self.case = case
        self.A, sizes = _matrix(case, seed)
        self.B = _rhs(self.A, _solution(self.A.shape[0], case["nrhs"], seed))
        self.solver = SymLDLT(torch.cuda.current_device())
        if case["kind"] in ("kkt", "ipm"):
            self.solver.setMode(Mode.StaticRegularized)
            self.solver.setKKTBlockSizes(*sizes)
            self.solver.setGraphLaunch(True)
        self.solver.analyzePattern(self.A)
        if case["kind"] == "grid2":
            self.solver.factorize(self.A)  # the pass refactorizes


class Batch:
    """Many systems as one batch (ma57_b200.batch)."""

    def __init__(self, case, seed):
        systems = _systems(case, seed)
        self.solver = BatchedSolver([S for S, _ in systems], device=torch.cuda.current_device())
        self.Bs = [_rhs(S, X) for S, X in systems]


def prepare(case, seed):
    if case["kind"] == "batch":
        return case, Batch(case, seed)
    return case, (DeviceSystem if case["kind"] in ("grid3", "solve") else HostSystem)(case, seed)


def run(state):
    case, s = state
    kind = case["kind"]
    if kind == "solve":
        return {"x": s.solve()}
    if kind == "grid3":
        return {"inertia": s.factorize(), "x": s.solve_refined()}
    if kind == "batch":
        s.solver.factorize()
        return {"x": np.concatenate(s.solver.solve(s.Bs)).T}
    if kind == "grid2":
        s.solver.refactorize(s.A)
        x = s.solver.solve(s.B)
    elif kind in ("kkt", "ties"):
        s.solver.factorize(s.A)
        x = s.solver.solveWithRefinement(s.A, s.B, RefinementOptions(tolerance=1e-12)).x
    else:
        s.solver.factorize(s.A)
        x = s.solver.solveWithGmresRefinement(s.A, s.B, GmresRefinementOptions(tolerance=1e-13)).x
    return {"inertia": np.array(s.solver.inertia().as_tuple()), "x": np.ascontiguousarray(x.T)}


def exact(case, seed):
    """The drawn solutions: B = A X is exact in 64 bits (see the top)."""
    if case["kind"] == "batch":
        return {"x": np.concatenate([X for _, X in _systems(case, seed)]).T}
    if case["kind"] in ("grid3", "solve"):
        n = case["k"] ** 3
    elif case["kind"] == "grid2":
        n = case["a"] * case["b"]
    elif case["kind"] == "ipm":
        n = case["k"] ** 3 + case["k"] ** 3 // 2
    else:
        n = case["grid"] ** 2 + case["n2"]
    x = np.ascontiguousarray(_solution(n, case["nrhs"], seed).T)
    return {"x": x} if case["kind"] == "solve" else {"inertia": None, "x": x}


# --------------------------------------------------------------------------
# Algorithmic work and tolerance


@functools.lru_cache(maxsize=64)
def _factor_size(key):
    """(nnz(L), factorization flops, nnz(A), n) of a pattern: columns of c_j
    entries, r = c_j - 1: r divisions and r (r + 1) multiply-adds."""
    case = dict(key)
    if case["kind"] == "batch":
        parts = []
        for i in range(case["count"]):
            S, _, _, _ = M.config4_system(i)
            n, cp, ri, _ = as_csc(S)
            parts.append((Analysis(n, cp, ri, OrderingType.AMD, SymbolicFactorOptions()), S.nnz))
    else:
        parts = [(_analysis(key), _matrix(case, 0)[0].nnz)]
    nnzl = flops = nnza = n = 0
    for an, nz in parts:
        c = an.factor().etree.colCount.astype(np.float64)
        nnzl, flops = nnzl + c.sum(), flops + ((c - 1) * (c + 1)).sum()
        nnza, n = nnza + nz, n + an.n
    return float(nnzl), float(flops), float(nnza), n


def work(case):
    """The factor written once and read twice (forward and backward solve),
    the values, right-hand sides and solutions once each. A refined solve
    cannot do without one solve and one residual."""
    key = (("kind", "batch"), ("count", case["count"])) if case["kind"] == "batch" else _pattern_key(case)
    nnzl, ff, nnza, n = _factor_size(key)
    r = case["nrhs"]
    vec = 16.0 * n * r
    solve_flops = 4.0 * nnzl * r
    if case["kind"] == "solve":
        return {"bytes": 16.0 * nnzl + vec, "flops": solve_flops}
    refined = case["kind"] not in ("grid2", "batch")
    return {"bytes": 24.0 * nnzl + 8.0 * nnza + vec + (8.0 * nnza if refined else 0.0),
            "flops": ff + solve_flops + (4.0 * nnza * r if refined else 0.0)}


# (rel, max), from the errors measured against the exact solutions over two
# seeds and about ten drawn cases of each kind; the largest seen follows
TOLERANCE = {
    "grid2": {"rel": 1e-10, "max": 1e-9},    # 3.3e-12, 1.9e-11
    "batch": {"rel": 5e-9, "max": 5e-7},     # 2.1e-10, 1.7e-8: the most singular of its random shifts
    "grid3": {"rel": 1e-10, "max": 1e-9},    # 1.8e-11, 4e-11
    "mixed": {"rel": 1e-8, "max": 1e-7},     # 1.6e-9, 1e-8: refined to 1e-12
    "solve": {"rel": 1e-10, "max": 1e-9},    # 4.1e-12, 3.9e-11
    "kkt": {"rel": 5e-9, "max": 1e-6},       # 5.2e-10, 6.4e-8: refined to 1e-12
    "ipm": {"rel": 1e-12, "max": 5e-11},     # 2.1e-14, 8.7e-13
    "ties": {"rel": 5e-14, "max": 5e-13},    # 1.2e-15, 6.0e-15
}


def tolerance(case):
    """The forward error of a backward-stable 64-bit solve is the system's
    condition number times 2^-53; the factor's rounding enters through the
    order of its sums. Unrefined batches and refinement that stops at a
    backward error of 1e-12 leave more."""
    return TOLERANCE[case["kind"] if case.get("precision") != "mixed" else "mixed"]
