// Panel factorization of large fronts under static pivoting
// (dense_kernel.hpp:919-1059): no pivot is rejected, interchanged or delayed,
// so a panel needs no agreement between the CTAs that share its rows, and
// panel `it` of a front always takes pivots 32 it, 32 it + 1, ...: which CTAs
// have rows, the panel's range and its outer block follow from the iteration's
// number and the front's sizes alone, not from the state that the launch
// rewrites. Each CTA with rows factors the panel's diagonal block for itself
// while its rows load, then eliminates one row per thread straight from and to
// global memory; the last of them to have read the block and the state (a
// ticket per front, no waiting) writes the diagonal block, D and the front's
// state.
//
// What bounds it is latency: the front's descriptor and state, the block, its
// LDL^T (one warp), a row pass of 496 multiply-adds. The cluster kernel that
// threshold pivoting uses kept the rows in the shared memory of at most 16
// CTAs, exchanged per-pivot maxima it did not need here, and had to narrow
// its panels on fronts of more than 10,000 rows: 33 us for 16 pivots of a
// 15568-row front, against 24 us for 32 here when this kernel was new (all
// panels of that KKT step: 33.0 and 12.2 ms, 10.9 now; an interior-point
// step's: 2.4 and 1.4 ms, 1.2 now).
#include <algorithm>

#include "common.cuh"
#include "factor_kernels.h"
#include "panel_block.cuh"
#include "reduce.cuh"

namespace symla_gpu {

namespace {
constexpr int kRowsPerCta = 96;  // one row per thread of warps 1 .. 3
constexpr int kStaticThreads = 32 + kRowsPerCta;
static_assert(kOuterBlock % kPanelMax == 0, "a panel never crosses an outer block");
}  // namespace

__global__ void __launch_bounds__(kStaticThreads, 2) static_panel_kernel(const FrontDesc* __restrict__ fronts,
                                                                      FrontState* st,
                                                                      const int* __restrict__ front_list,
                                                                      KernelOpts o, FactorGlobals* g, int level,
                                                                      int dynamic, int it) {
  if (level_skipped(g, level, dynamic)) return;
  __shared__ __align__(16) DiagBlock B;
  __shared__ double s_max[kStaticThreads / 32];
  __shared__ int s_last;
  const int s = front_list[blockIdx.y];
  const FrontDesc f = fronts[s];
  const int m = f.m, tile = blockIdx.x;
  const int ps = it * kPanelMax;
  if (it > 0 && ps >= f.nelig) {
    // finished by an earlier panel: the updates that follow must do nothing
    if (tile == 0 && threadIdx.x == 0) {
      st[s].panel_start = f.nelig;
      st[s].far = 0;
    }
    return;
  }
  const int ob = ps - ps % kOuterBlock, ob_end = min(ob + kOuterBlock, f.nelig);
  const int pe = min(ps + kPanelMax, ob_end), np = pe - ps;
  const int ntiles = max(1, (m - pe + kRowsPerCta - 1) / kRowsPerCta);
  if (tile >= ntiles) return;
  // all that is read of the state before the ticket (the running maximum,
  // which the other CTAs raise, is not)
  double om = st[s].orig_max, delta = st[s].delta, tmax = 0.0;
  if (ps == 0) {
    // first panel: max |entry| of the assembled front, from the assembly kernel
    if (om < o.static_abs_floor) om = 1.0;
    tmax = om;
    delta = o.front_delta ? o.front_delta[s] : (o.static_delta > 0.0 ? o.static_delta : 1.4901161193847656e-08 * om);
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t ld = f.ld;
  double* F = f.F;
  const int i = pe + tile * kRowsPerCta + static_cast<int>(threadIdx.x) - 32;
  const bool row = warp > 0 && i < m;
  double a[kPanelMax];
  if (warp == 0) {
    const int sign = (o.sign_final && lane < np) ? o.sign_final[f.fidx[ps + lane]] : 0;
    const double floorv = fmax(o.static_abs_floor, o.static_rel_floor * om);
    // the loads of all columns first: they must not wait for one another's stores
    double v[kPanelMax];
#pragma unroll
    for (int j = 0; j < kPanelMax; ++j)
      v[j] = (lane >= j && lane < np) ? F[static_cast<int64_t>(ps + j) * ld + ps + lane] : 0.0;
#pragma unroll
    for (int j = 0; j < kPanelMax; ++j) B.db[lane][j] = v[j];
    __syncwarp();
    if (factor_diag_block<true>(B, np, lane, sign, floorv, delta)) {
#pragma unroll 1
      for (int j = 0; j < np; ++j)
        B.db[lane][j] = (lane >= j && lane < np) ? F[static_cast<int64_t>(ps + j) * ld + ps + lane] : 0.0;
      factor_diag_block_divide<true>(B, np, lane, sign, floorv, delta);
    }
  } else {
#pragma unroll
    for (int c = 0; c < kPanelMax; ++c) a[c] = (row && c < np) ? F[static_cast<int64_t>(ps + c) * ld + i] : 0.0;
  }
  __syncthreads();
  // The CTA has read the block and the state. Taken here, with no stores of the
  // CTA outstanding, the fence costs nothing; after the rows' it took 2.3 us.
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(&st[s].ticket, 1) == ntiles - 1;
    __threadfence();
  }
  if (row) {
    panel_row(B, np, a);
    double* out = F + static_cast<int64_t>(ps) * ld + i;
    store_panel_row(B, np, a, f.P, f.pw, f.prt, ps - ob, i,
                    [&](int c, double l) { out[static_cast<int64_t>(c) * ld] = l; });
#pragma unroll
    for (int c = 0; c < kPanelMax; ++c)
      if (c < np) tmax = fmax(tmax, fabs(a[c]));
  } else if (warp == 0 && lane < np) {
    // the block's own values
    double v = fabs(B.dv[lane]);
    for (int r = lane + 1; r < np; ++r) v = fmax(v, fabs(B.wv[r][lane]));
    tmax = fmax(tmax, v);
  }
  tmax = warp_max(tmax);
  if (lane == 0) s_max[warp] = tmax;
  const bool done = pe >= f.nelig;
  if (done)
    for (int t = tile * kStaticThreads + threadIdx.x; t < m; t += ntiles * kStaticThreads) f.lpos[f.lperm[t]] = t;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kStaticThreads / 32; ++w) tmax = fmax(tmax, s_max[w]);
    atomic_max_nonneg(&st[s].running_max, tmax);
  }
  if (!s_last) return;
  // every CTA of the front has read the block and the state: they are this one's to write
  for (int t = threadIdx.x; t < np * np; t += kStaticThreads) {
    const int c = t / np, r = t % np;
    if (r >= c) F[static_cast<int64_t>(ps + c) * ld + ps + r] = B.db[r][c];
  }
  if (warp == 0) {
    const bool in = lane < np;
    const double d = in ? B.dv[lane] : 0.0;
    if (in) {
      f.Dd[ps + lane] = d;
      f.Do[ps + lane] = 0.0;
      f.pk[ps + lane] = 0;
    }
    const unsigned pos = __ballot_sync(0xffffffffu, in && d > 0);
    const unsigned neg = __ballot_sync(0xffffffffu, in && d < 0);
    const unsigned zer = __ballot_sync(0xffffffffu, in && !(d > 0) && !(d < 0));
    const unsigned per = __ballot_sync(0xffffffffu, in && B.pv[lane] != 0.0);
    if (lane == 0) {
      const bool first = ps == 0;
      FrontState& W = st[s];
      double pert = first ? 0.0 : W.perturb;
      for (int c = 0; c < np; ++c)  // in pivot order
        if (per >> c & 1) pert += fabs(B.pv[c]);
      W.orig_max = om;
      W.delta = delta;
      W.n_pos = (first ? 0 : W.n_pos) + __popc(pos);
      W.n_neg = (first ? 0 : W.n_neg) + __popc(neg);
      W.n_zero = (first ? 0 : W.n_zero) + __popc(zer);
      W.num_perturbed = (first ? 0 : W.num_perturbed) + __popc(per);
      W.perturb = pert;
      W.panel_start = ps;
      W.k = pe;
      W.npiv = pe;
      W.ob = ob;
      W.ob_end = ob_end;
      W.far = (done || pe >= ob_end) ? 1 : 0;
      W.ticket = 0;
      int flags = 0;
      if (done) {
        flags = kFlagDone;
        if (pe < m && f.parent < 0) flags |= kFlagSingularRoot;
      }
      W.flags = flags;
      atomicAdd(&g->spec_full, 1);
    }
  }
}

void launch_static_panel(const FrontDesc* fronts, FrontState* st, const int* list, int count, int max_m,
                         const KernelOpts& o, FactorGlobals* g, int level, int dynamic, int it, cudaStream_t stream) {
  if (count <= 0) return;
  const int tiles = std::max(1, (max_m + kRowsPerCta - 1) / kRowsPerCta);
  for (int b = 0; b < count; b += 65535)  // grid.y limit
    static_panel_kernel<<<dim3(tiles, std::min(count - b, 65535)), kStaticThreads, 0, stream>>>(
        fronts, st, list + b, o, g, level, dynamic, it);
}

}  // namespace symla_gpu
