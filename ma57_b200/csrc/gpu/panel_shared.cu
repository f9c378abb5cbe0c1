// Panel of up to NB pivots of a large front by one CTA, pivot by pivot
// (dense_kernel.hpp:516-793), for fronts of at most kPanelSharedRows rows:
// thread t owns rows t, t + NT, ..., the panel's L stays in shared memory
// beside the front, and the candidate column's values in registers.
//
// What bounds it is the latency of a pivot's steps: the column's sums over the
// panel's pivots, the argmax over the block, the store of L. Each warp forms
// D L(k, :) for itself, the argmax is three 32-bit reductions on either side
// of its barrier, a quotient is three multiply-adds on 1 / d, and the next column's values are loaded
// a step ahead, so a plain 1x1 pivot takes two block barriers. The general
// single-CTA panel (factor_kernels.cu), which reads L back from global memory
// and forms every quotient, took 94 us for 32 plain pivots of 693 rows and 64
// of 229, against 68 and 43 us here; the panels of a 20^3 7-point grid (which
// decide about seven pivots of a panel by the second test) 4.6 and 3.1 ms.
#include <algorithm>

#include "common.cuh"
#include "factor_kernels.h"
#include "panel_block.cuh"
#include "reduce.cuh"

namespace symla_gpu {

namespace {
constexpr double kAlphaBK = 0.64038820320220756;  // (1 + sqrt(17)) / 8
constexpr int kCols = kPanelWidth + 2;            // a 2x2 pivot may pass the panel's end
}  // namespace

template <int NT, int R>
__global__ void __launch_bounds__(NT) panel_shared_kernel(const FrontDesc* __restrict__ fronts, FrontState* st,
                                                          const int* __restrict__ front_list, int nb, KernelOpts o,
                                                          FactorGlobals* g, int level, int dynamic) {
  if (level_skipped(g, level, dynamic)) return;
  constexpr int NW = NT / 32;
  extern __shared__ __align__(16) double smem[];
  __shared__ double wv[NW][kPanelWidth];  // D L(col, :)^T, a copy per warp
  __shared__ double sDd[kCols], sDo[kCols];
  __shared__ int spk[kCols];
  __shared__ double arg_v[NW], max_v[NW], rm_v[NW];
  __shared__ int arg_i[NW];

  const int s = front_list[blockIdx.x];
  const FrontDesc f = fronts[s];
  FrontState S = st[s];
  if (S.flags & kFlagDone) {
    // no panel in this iteration: the updates that follow must do nothing
    if (threadIdx.x == 0) {
      st[s].panel_start = S.k;
      st[s].far = 0;
    }
    return;
  }
  if (S.ob_end == 0 || S.far) {
    S.ob = S.k;
    S.ob_end = min(S.k + kOuterBlock, f.nelig);
    S.far = 0;
  }
  const int m = f.m, effEnd = f.nelig;
  const int64_t ld = f.ld;
  double* F = f.F;
  double* L = smem;                 // L(i, q) at L[q m + i]
  double* colk = smem + kCols * m;  // the candidate column and its partner
  double* colr = colk + m;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  // first panel: orig_max of the assembled front (from the assembly kernel)
  if (S.k == 0) {
    double om = S.orig_max;
    if (om < (o.mode == 1 ? o.static_abs_floor : o.zero_tol)) om = 1.0;
    S.orig_max = om;
    S.running_max = om;
    S.n_pos = S.n_neg = S.n_zero = 0;
    S.num_perturbed = 0;
    S.perturb = 0.0;
    S.delta = o.front_delta ? o.front_delta[s] : (o.static_delta > 0.0 ? o.static_delta : 1.4901161193847656e-08 * om);
  }
  const double orig_max = S.orig_max;
  const int ps = S.k, pe = ps + min(nb, S.ob_end - ps);
  int k = ps;
  double rmax = 0.0;  // running max of this thread's rows
  bool stopped = false, flush = false;

  // raw values of column col, rows >= k, of this thread's rows
  auto load_raw = [&](int col, int from, double (&raw)[R]) {
#pragma unroll
    for (int n = 0; n < R; ++n) {
      const int i = tid + n * NT;
      raw[n] = (i < from || i >= m) ? 0.0 : (i >= col ? F[col * ld + i] : F[i * ld + col]);
    }
  };
  // v = raw - L (D L(col, :)^T) over the panel's p pivots
  auto column = [&](int col, int p, const double (&raw)[R], double (&v)[R]) {
    double* w = wv[warp];
    if (lane < p) {
      const int kind = spk[lane];
      double x = sDd[lane] * L[lane * m + col];
      if (kind == 1) x += sDo[lane] * L[(lane + 1) * m + col];
      if (kind == 2) x += sDo[lane - 1] * L[(lane - 1) * m + col];
      w[lane] = x;
    }
    __syncwarp();
    double c0[R], c1[R];
#pragma unroll
    for (int n = 0; n < R; ++n) c0[n] = c1[n] = 0.0;
    const double* l = L + tid;
    int q = 0;
    for (; q + 4 <= p; q += 4, l += 4 * m) {
      const double w0 = w[q], w1 = w[q + 1], w2 = w[q + 2], w3 = w[q + 3];
#pragma unroll
      for (int n = 0; n < R; ++n)
        if (tid + n * NT < m) {
          c0[n] = fma(l[n * NT], w0, c0[n]);
          c1[n] = fma(l[n * NT + m], w1, c1[n]);
          c0[n] = fma(l[n * NT + 2 * m], w2, c0[n]);
          c1[n] = fma(l[n * NT + 3 * m], w3, c1[n]);
        }
    }
    for (; q < p; ++q, l += m)
#pragma unroll
      for (int n = 0; n < R; ++n)
        if (tid + n * NT < m) c0[n] = fma(l[n * NT], w[q], c0[n]);
#pragma unroll
    for (int n = 0; n < R; ++n) v[n] = raw[n] - (c0[n] + c1[n]);
    __syncwarp();  // w is the warp's next column's
  };
  // L and -(L D) of pivot kk, row i, to shared memory, the front and the
  // packed operands of the updates
  auto put = [&](int kk, int i, double l, double a) {
    L[(kk - ps) * m + i] = l;
    F[kk * ld + i] = l;
    double* pk = f.P + packed_at(f.prt, kk - S.ob, i);
    pk[0] = l;
    pk[f.pw] = -a;
  };
  auto set_d = [&](int kk, double dd, double doff, int kind) {
    sDd[kk - ps] = dd;
    sDo[kk - ps] = doff;
    spk[kk - ps] = kind;
    f.Dd[kk] = dd;
    f.Do[kk] = doff;
    f.pk[kk] = static_cast<int8_t>(kind);
    F[kk * ld + kk] = dd;
  };
  auto count = [&](double d) {
    if (d > 0)
      ++S.n_pos;
    else if (d < 0)
      ++S.n_neg;
    else
      ++S.n_zero;
  };
  // symmetric interchange of positions a < b: the front, its indices, the
  // packed rows of the outer block's pivots and the panel's L. Ends in a
  // barrier.
  auto interchange = [&](int a, int b) {
    auto swap = [](double& x, double& y) {
      const double t = x;
      x = y;
      y = t;
    };
    for (int t = tid; t < m - 1; t += NT) {
      if (t < a)
        swap(F[t * ld + a], F[t * ld + b]);
      else if (t < b - 1)
        swap(F[a * ld + t + 1], F[(t + 1) * ld + b]);
      else if (t == b - 1)
        swap(F[a * ld + a], F[b * ld + b]);
      else
        swap(F[a * ld + t + 1], F[b * ld + t + 1]);
    }
    for (int t = tid; t < k - S.ob; t += NT) {
      double* pa = f.P + packed_at(f.prt, t, a);
      double* pb = f.P + packed_at(f.prt, t, b);
      swap(pa[0], pb[0]);
      swap(pa[f.pw], pb[f.pw]);
    }
    if (tid < k - ps) swap(L[tid * m + a], L[tid * m + b]);
    if (tid == 0) {
      int x = f.fidx[a];
      f.fidx[a] = f.fidx[b];
      f.fidx[b] = x;
      x = f.lperm[a];
      f.lperm[a] = f.lperm[b];
      f.lperm[b] = x;
    }
    __syncthreads();
  };
  // 1x1 pivot d at k from the column values v
  auto finish_1x1 = [&](double d, const double (&v)[R]) {
    count(d);
    rmax = fmax(rmax, fabs(d));
    const double inv = pivot_reciprocal(d);
    const bool extreme = pivot_extreme(d);
#pragma unroll
    for (int n = 0; n < R; ++n) {
      const int i = tid + n * NT;
      if (i > k && i < m) {
        rmax = fmax(rmax, fabs(v[n]));
        put(k, i, pivot_quotient(v[n], d, inv, extreme), v[n]);
      }
    }
    if (tid == 0) set_d(k, d, 0.0, 0);
    __syncthreads();
    ++k;
  };

  double raw[R], v[R], u[R];
  int raw_col = -1;  // the column raw holds
  while (k < pe) {
    const int p = k - ps;
    if (raw_col != k) load_raw(k, k, raw);
    column(k, p, raw, v);
#pragma unroll
    for (int n = 0; n < R; ++n) {
      const int i = tid + n * NT;
      if (i >= k && i < m) colk[i] = v[n];
    }
    raw_col = -1;
    if (k + 1 < pe) {
      load_raw(k + 1, k + 1, raw);
      raw_col = k + 1;
    }
    if (o.mode == 1) {
      __syncthreads();
      double applied;
      const double d = static_pivot(colk[k], o.sign_final ? o.sign_final[f.fidx[k]] : 0,
                                    fmax(o.static_abs_floor, o.static_rel_floor * orig_max), S.delta, applied);
      if (applied != 0.0) {
        S.perturb += fabs(applied);
        ++S.num_perturbed;
      }
      finish_1x1(d, v);
      continue;
    }
    ArgMax am{0.0, -1};
#pragma unroll
    for (int n = 0; n < R; ++n) {
      const int i = tid + n * NT;
      if (i > k && i < effEnd) am = argmax_combine(am, ArgMax{fabs(v[n]), i});
    }
    am = warp_argmax_nonneg(am);
    if (lane == 0) {
      arg_v[warp] = am.v;
      arg_i[warp] = am.i;
    }
    __syncthreads();
    am = warp_argmax_nonneg(lane < NW ? ArgMax{arg_v[lane], arg_i[lane]} : ArgMax{0.0, -1});
    const double lambda = am.v, akk = colk[k];
    const int r = am.i;
    int dec;  // 0: 1x1 at k, 1: interchange k <-> r, 1x1, 2: 2x2 (k, r), 3: stop, 4: flush
    double arr = 0.0, vkr = 0.0;
    if (lambda <= o.zero_tol) {
      const double isolatedFloor = fmax(o.zero_tol, o.rel_floor * orig_max);
      dec = (fabs(akk) <= isolatedFloor) ? 3 : 0;
    } else if (r < 0 || fabs(akk) >= kAlphaBK * lambda) {  // (r < 0: no candidate, under a negative zero_tol)
      dec = 0;
    } else if (r >= S.ob_end && ps > S.ob) {
      dec = 4;  // partner beyond the outer block: apply the deferred update first
    } else {
      double rr[R];
      load_raw(r, k, rr);
      column(r, p, rr, u);
      double smax = 0.0;
#pragma unroll
      for (int n = 0; n < R; ++n) {
        const int i = tid + n * NT;
        if (i >= k && i < m) {
          colr[i] = u[n];
          if (i < effEnd && i != r) smax = fmax(smax, fabs(u[n]));
        }
      }
      smax = warp_max_nonneg(smax);
      if (lane == 0) max_v[warp] = smax;
      __syncthreads();
      const double sigma = warp_max_nonneg(lane < NW ? max_v[lane] : 0.0);
      arr = colr[r];
      vkr = colk[r];
      if (fabs(akk) * sigma >= kAlphaBK * lambda * lambda)
        dec = 0;
      else if (fabs(arr) >= kAlphaBK * sigma)
        dec = 1;
      else
        dec = 2;
    }
    if (dec == 3) {
      stopped = true;
      break;
    }
    if (dec == 4) {
      flush = true;
      break;
    }
    if (dec == 0) {
      finish_1x1(akk, v);
      continue;
    }
    raw_col = -1;  // an interchange moves the raw values, a 2x2 pivot takes the next column
    if (dec == 1) {
      // the new column k is column r with rows k and r exchanged
#pragma unroll
      for (int n = 0; n < R; ++n)
        if (tid + n * NT == r) u[n] = colr[k];
      interchange(k, r);
      finish_1x1(arr, u);
      continue;
    }
    // 2x2: bring r to k + 1
    const double d11 = akk, d21 = vkr, d22 = arr;
    const double det = d11 * d22 - d21 * d21;
    rmax = warp_max_nonneg(rmax);
    if (lane == 0) rm_v[warp] = rmax;
    if (r != k + 1) {
#pragma unroll
      for (int n = 0; n < R; ++n)
        if (tid + n * NT == r) {
          v[n] = colk[k + 1];
          u[n] = colr[k + 1];
        }
      interchange(k + 1, r);
    } else {
      __syncthreads();
    }
    const double rm1 = fmax(1.0, fmax(S.running_max, warp_max_nonneg(lane < NW ? rm_v[lane] : 0.0)));
    if (fabs(det) <= o.zero_tol * rm1 * rm1) {
      stopped = true;
      break;
    }
    rmax = fmax(rmax, fmax(fabs(d11), fmax(fabs(d21), fabs(d22))));
    if (det < 0) {
      ++S.n_pos;
      ++S.n_neg;
    } else {
      const double tr = d11 + d22;
      if (tr > 0)
        S.n_pos += 2;
      else if (tr < 0)
        S.n_neg += 2;
      else {
        ++S.n_pos;
        ++S.n_neg;
      }
    }
    const double inv11 = d22 / det, inv21 = -d21 / det, inv22 = d11 / det;
#pragma unroll
    for (int n = 0; n < R; ++n) {
      const int i = tid + n * NT;
      if (i >= k + 2 && i < m) {
        rmax = fmax(rmax, fmax(fabs(v[n]), fabs(u[n])));
        put(k, i, v[n] * inv11 + u[n] * inv21, v[n]);
        put(k + 1, i, v[n] * inv21 + u[n] * inv22, u[n]);
      }
    }
    if (tid == 0) {
      set_d(k, d11, d21, 1);
      set_d(k + 1, d22, 0.0, 2);
      F[k * ld + k + 1] = d21;
    }
    __syncthreads();
    k += 2;
  }

  rmax = warp_max_nonneg(rmax);
  __syncthreads();
  if (lane == 0) rm_v[warp] = rmax;
  if (stopped || k >= effEnd)
    for (int t = tid; t < m; t += NT) f.lpos[f.lperm[t]] = t;
  __syncthreads();
  if (tid == 0) {
    for (int w = 0; w < NW; ++w) rmax = fmax(rmax, rm_v[w]);
    FrontState& W = st[s];
    W.orig_max = orig_max;
    W.delta = S.delta;
    W.running_max = fmax(S.running_max, rmax);
    W.n_pos = S.n_pos;
    W.n_neg = S.n_neg;
    W.n_zero = S.n_zero;
    W.num_perturbed = S.num_perturbed;
    W.perturb = S.perturb;
    W.panel_start = ps;
    W.k = k;
    W.npiv = k;
    W.ob = S.ob;
    W.ob_end = S.ob_end;
    W.far = (stopped || k >= effEnd || flush || k >= S.ob_end) ? 1 : 0;
    int flags = flush ? kFlagFlush : 0;
    if (stopped || k >= effEnd) {
      flags |= kFlagDone;
      if (k < effEnd) {
        if (f.parent >= 0) {
          flags |= kFlagDelayed;
          atomicMin(&g->delay_level, f.level);
        } else {
          flags |= kFlagSingularRoot;
        }
      } else if (k < m && f.parent < 0) {
        flags |= kFlagSingularRoot;
      }
    }
    W.flags = flags;
  }
}

namespace {
size_t shared_panel_smem(int max_m) { return static_cast<size_t>(kCols + 2) * max_m * sizeof(double); }
constexpr int kSmallRows = 256;
}  // namespace

cudaError_t configure_shared_panel() {
  const cudaError_t e = cudaFuncSetAttribute(panel_shared_kernel<kSmallRows, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             static_cast<int>(shared_panel_smem(kSmallRows)));
  if (e != cudaSuccess) return e;
  static_assert(kPanelSharedRows <= 2 * 512);
  return cudaFuncSetAttribute(panel_shared_kernel<512, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              static_cast<int>(shared_panel_smem(kPanelSharedRows)));
}

cudaError_t launch_shared_panel(const FrontDesc* fronts, FrontState* st, const int* list, int count, int max_m, int nb,
                                const KernelOpts& o, FactorGlobals* g, int level, int dynamic, cudaStream_t stream) {
  if (count <= 0) return cudaSuccess;
  if (max_m > kPanelSharedRows || nb > kPanelWidth) return cudaErrorInvalidValue;
  if (max_m <= kSmallRows)
    panel_shared_kernel<kSmallRows, 1><<<count, kSmallRows, shared_panel_smem(max_m), stream>>>(fronts, st, list, nb, o,
                                                                                                g, level, dynamic);
  else
    panel_shared_kernel<512, 2><<<count, 512, shared_panel_smem(max_m), stream>>>(fronts, st, list, nb, o, g, level,
                                                                                  dynamic);
  return cudaGetLastError();
}

}  // namespace symla_gpu
