"""Front-size-to-tile-shape schedule chosen by measurement.

Two launch shapes depend on front size and have no single best value: the
number of CTAs in the panel cluster of the large fronts (2, 4, 8 or 16; more
CTAs hold fewer rows each but occupy more SMs; or 1, the single-CTA panel
kernel, whose pivot-by-pivot decisions need no cluster barriers) and the
tile shape of their Schur-complement update (128 x 64 or 64 x 64: the smaller
tile wastes less of small fronts' trailing blocks, the larger reuses operands
more). Under static pivoting, whose panels use no clusters, only 1 differs from
the default. The tree levels are bucketed by the largest front they hold, and a coordinate search times the actual
factorization (CUDA events around the numeric factorization) for each
candidate shape of one bucket at a time, keeping the fastest. The result is
installed per level through symla_gpu_set_level_schedule; it changes launch
shapes only, and results by no more than rounding.
"""
from __future__ import annotations

import ctypes as C
import math

from . import _lib as L
from .solver import Mode

LARGE_BUCKETS = (512, 2048, 8192, 1 << 30)  # panel cluster, by the level's largest large front


def level_info(solver):
    """Per level: small/large front counts and largest sizes, and the
    installed shapes."""
    lib = L.load()
    h = solver._ctx.h
    nlev = int(solver.plan_stats()["levels"])
    out = []
    buf = (C.c_int * 6)()
    for lv in range(nlev):
        if lib.symla_gpu_level_info(h, lv, buf) != L.SYMLA_OK:
            raise RuntimeError(L.last_error())
        out.append({"small": buf[0], "small_max_m": buf[1], "large": buf[2], "large_max_m": buf[3],
                    "small_threads": buf[4], "cluster_ctas": buf[5]})
    return out


def _bucket(value, edges):
    for i, e in enumerate(edges):
        if value <= e:
            return i
    return len(edges) - 1


def apply(solver, schedule):
    """schedule: {"small": {}, "large": {bucket: ctas}, "update": {bucket:
    tile rows}} (missing entries: the default shape; small fronts take their
    kernel by size)."""
    lib = L.load()
    for lv, info in enumerate(level_info(solver)):
        lb = _bucket(info["large_max_m"], LARGE_BUCKETS)
        cl = schedule["large"].get(lb, 0) if info["large"] else 0
        ur = schedule.get("update", {}).get(lb, 0) if info["large"] else 0
        if lib.symla_gpu_set_level_schedule(solver._ctx.h, lv, 0, cl) != L.SYMLA_OK:
            raise RuntimeError(L.last_error())
        if lib.symla_gpu_set_level_update_rows(solver._ctx.h, lv, ur) != L.SYMLA_OK:
            raise RuntimeError(L.last_error())


def _factor_ms(solver, A, reps):
    best = math.inf
    for _ in range(reps):
        solver.factorize(A)
        best = min(best, solver.phase_ms()[6])
    return best


def tune(solver, A, reps: int = 2):
    """Coordinate search over the buckets present in `solver`'s plan (the
    pattern of A must be analyzed and factorized once). Returns the chosen
    schedule (installed) and the measured default / tuned factorization ms."""
    info = level_info(solver)
    large_b = sorted({_bucket(i["large_max_m"], LARGE_BUCKETS) for i in info if i["large"]})
    schedule = {"small": {}, "large": {}, "update": {}}
    apply(solver, schedule)
    base = _factor_ms(solver, A, reps)
    best = base
    panels = (1,) if solver.mode_ == Mode.StaticRegularized else (1, 2, 4, 8, 16)
    for kind, buckets, cands in (("large", large_b, panels), ("update", large_b, (64, 128))):
        for b in buckets:
            for cand in cands:
                trial = {k: dict(v) for k, v in schedule.items()}
                trial[kind][b] = cand
                apply(solver, trial)
                t = _factor_ms(solver, A, reps)
                if t < best:
                    best, schedule = t, trial
    apply(solver, schedule)
    return schedule, base, best
