// Fronts of at most kSmallFrontMax rows, one CTA per front: assembly
// (multifrontal.hpp:498-535), threshold Bunch-Kaufman (dense_kernel.hpp:
// 576-793) or static pivoting (:919-1059) and write-back in one launch, the
// front's lower triangle in shared memory. (Fronts of at most 32 rows in
// numbers take a warp each, factor_small_kernel.)
//
// Thread t owns row t. Pivots go in panels of 16: the candidate column is
// brought up to date from the panel's L and its columns before scaling
// (W = L D), decided, and stored; the rest of the front is updated once per
// panel on the FP64 tensor path. What bounds it is the latency of a pivot's
// steps: sums over at most 16 pivots, an argmax of three 32-bit reductions on
// either side of a block barrier, the store of L, a second barrier. Updating
// the whole front after every pivot with 256 threads took 2.0 ms for the 11
// levels of a 53 x 74 grid and 2.36 ms for the small fronts of a 64^3 27-point
// grid, now 0.9 and 0.7 ms.
#include <algorithm>

#include "common.cuh"
#include "factor_kernels.h"
#include "panel_block.cuh"
#include "reduce.cuh"

namespace symla_gpu {

namespace {
constexpr double kAlphaBK = 0.64038820320220756;  // (1 + sqrt(17)) / 8
constexpr int kNT = 128;                          // threads = rows at most
static_assert(kSmallFrontMax <= kNT);
constexpr int kNB = 16;          // pivots per panel (one more when a 2x2 ends it)
constexpr int kWS = 140;         // stride of the panel's W rows: conflict-free fragments, 8 columns past the front
constexpr int kBatch = 32;       // children whose descriptors are staged at a time

// leading dimension of the front in shared memory: conflict-free fragments
__host__ __device__ inline int front_lds(int m) { return ((m + 15) & ~15) + 4; }

__device__ __forceinline__ void small_dmma(double* c, const double* a, const double* b) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
               : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}
}  // namespace

__global__ void __launch_bounds__(kNT) small_front_kernel(const FrontDesc* __restrict__ fronts,
                                                          const ChildLink* __restrict__ links, FrontState* st,
                                                          const int* __restrict__ front_list,
                                                          const int* __restrict__ a_colptr, KernelOpts o,
                                                          FactorGlobals* g, int level, int dynamic) {
  if (level_skipped(g, level, dynamic)) return;
  constexpr int NW = kNT / 32;
  extern __shared__ __align__(16) double smem[];
  __shared__ const double* s_cb[kBatch];
  __shared__ int64_t s_cld[kBatch];
  __shared__ const int* s_rel[kBatch];
  __shared__ int s_ncb[kBatch];
  __shared__ int rel[2][kNT];
  __shared__ double colk[kNT], colr[kNT];
  __shared__ int fi[kNT], lp[kNT], sgn[kNT];
  __shared__ double arg_v[NW], max_v[NW], rm_v[NW];
  __shared__ int arg_i[NW];

  const int s = front_list[blockIdx.x];
  const FrontDesc f = fronts[s];
  const int m = f.m, lds = front_lds(m), effEnd = f.nelig;
  double* S = smem;                                   // S(i, j), i >= j, at S[j lds + i]
  double* W = smem + static_cast<size_t>(lds) * m;    // W(q, j) of the panel's pivots at W[q kWS + j]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  // ---- assembly: the children's contribution blocks in their fixed order,
  // then A's entries. A child's rows go to as many thread groups as fit.
  for (int t = tid; t < lds * m; t += kNT) S[t] = 0.0;
  if (tid < m) {
    fi[tid] = f.fidx[tid];
    lp[tid] = tid;
  }
  for (int b0 = f.ch_begin; b0 < f.ch_end; b0 += kBatch) {
    const int nb = min(kBatch, f.ch_end - b0);
    __syncthreads();
    if (tid < nb) {
      const ChildLink L = links[b0 + tid];
      const FrontDesc& cf = fronts[L.child];
      const int np = st[L.child].npiv;
      // the contribution block: L.cb rows from npiv (checked build: as many as there are)
      const bool ok = check(np >= 0 && np + L.cb <= cf.m, o.chk, kChkGather, L.child);
      s_cb[tid] = cf.F + static_cast<int64_t>(np) * cf.ld + np;
      s_cld[tid] = cf.ld;
      s_rel[tid] = L.relmap;
      s_ncb[tid] = ok ? L.cb : 0;
    }
    __syncthreads();
    int next = tid < s_ncb[0] ? s_rel[0][tid] : 0;
    for (int c = 0; c < nb; ++c) {
      const int cb = s_ncb[c];
      int* rc = rel[c & 1];
      rc[tid] = next;
      if (c + 1 < nb) next = tid < s_ncb[c + 1] ? s_rel[c + 1][tid] : 0;
      __syncthreads();  // (also: the previous child is added, its rows of rel are free)
      const int rows = (cb + 31) & ~31, groups = rows > 0 ? kNT / rows : 0;
      const int r = groups > 0 ? tid % rows : 0, grp = groups > 0 ? tid / rows : 0;
      if (r < cb && grp < groups) {
        const double* src = s_cb[c] + r;
        const int64_t ld = s_cld[c];
        const int pr = rc[r];
        for (int cc = grp; cc <= r; cc += 8 * groups) {
          double v[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) v[q] = cc + q * groups <= r ? src[(cc + q * groups) * ld] : 0.0;
#pragma unroll
          for (int q = 0; q < 8; ++q)
            if (cc + q * groups <= r) {
              const int pc = rc[cc + q * groups];
              S[min(pr, pc) * lds + max(pr, pc)] += v[q];
            }
        }
      }
    }
  }
  __syncthreads();
  {
    const int e0 = a_colptr[f.a_begin], e1 = a_colptr[f.a_begin + f.ncols];
    for (int e = e0 + tid; e < e1; e += kNT) {
      int j, i, idx;
      if (a_entry(o, f, e, j, i, idx)) S[j * lds + i] += o.values[idx];
    }
  }
  const bool is_static = o.mode == 1;
  if (is_static && tid < m) sgn[tid] = o.sign_final ? o.sign_final[fi[tid]] : 0;
  __syncthreads();

  // ---- orig_max over the whole front (dense_kernel.hpp:413, :934)
  double rmax = 0.0;  // running max of this thread's rows
  if (tid < m)
#pragma unroll 8
    for (int j = 0; j <= tid; ++j) rmax = fmax(rmax, fabs(S[j * lds + tid]));
  rmax = warp_max_nonneg(rmax);
  if (lane == 0) rm_v[warp] = rmax;
  __syncthreads();
  double orig_max = warp_max_nonneg(lane < NW ? rm_v[lane] : 0.0);
  if (orig_max < (is_static ? o.static_abs_floor : o.zero_tol)) orig_max = 1.0;
  const double delta =
      !is_static ? 0.0
                 : (o.front_delta ? o.front_delta[s]
                                  : (o.static_delta > 0.0 ? o.static_delta : 1.4901161193847656e-08 * orig_max));
  const double floorv = fmax(o.static_abs_floor, o.static_rel_floor * orig_max);
  rmax = 0.0;

  int n_pos = 0, n_neg = 0, n_zero = 0, nPert = 0;
  double pert = 0.0;
  int k = 0;
  bool stopped = false;
  while (k < effEnd && !stopped) {
    const int ks = k, pend = min(k + kNB, effEnd);
    // raw value minus the panel's pivots so far, for this thread's row
    auto column = [&](int col, double raw) {
      const int p = k - ks;
      const double* l = S + ks * lds + tid;
      const double* w = W + col;
      double c0 = 0.0, c1 = 0.0;
      int q = 0;
      for (; q + 4 <= p; q += 4, l += 4 * lds, w += 4 * kWS) {
        c0 = fma(l[0], w[0], c0);
        c1 = fma(l[lds], w[kWS], c1);
        c0 = fma(l[2 * lds], w[2 * kWS], c0);
        c1 = fma(l[3 * lds], w[3 * kWS], c1);
      }
      for (; q < p; ++q, l += lds, w += kWS) c0 = fma(l[0], w[0], c0);
      return raw - (c0 + c1);
    };
    // symmetric interchange of positions a < b (raw front, L, the panel's W);
    // ends in a barrier
    auto interchange = [&](int a, int b) {
      auto swap = [](double& x, double& y) {
        const double t = x;
        x = y;
        y = t;
      };
      const int t = tid;
      if (t < m - 1) {
        if (t < a)
          swap(S[t * lds + a], S[t * lds + b]);
        else if (t < b - 1)
          swap(S[a * lds + t + 1], S[(t + 1) * lds + b]);
        else if (t == b - 1)
          swap(S[a * lds + a], S[b * lds + b]);
        else
          swap(S[a * lds + t + 1], S[b * lds + t + 1]);
      }
      if (t < k - ks) swap(W[t * kWS + a], W[t * kWS + b]);
      if (t == 0) {
        int x = fi[a];
        fi[a] = fi[b];
        fi[b] = x;
        x = lp[a];
        lp[a] = lp[b];
        lp[b] = x;
      }
      __syncthreads();
    };
    auto finish_1x1 = [&](double d, double v) {
      if (d > 0)
        ++n_pos;
      else if (d < 0)
        ++n_neg;
      else
        ++n_zero;
      rmax = fmax(rmax, fabs(d));
      const double inv = pivot_reciprocal(d);
      const bool extreme = pivot_extreme(d);
      if (tid > k && tid < m) {
        rmax = fmax(rmax, fabs(v));
        S[k * lds + tid] = pivot_quotient(v, d, inv, extreme);
        W[(k - ks) * kWS + tid] = v;
      } else if (tid == k) {
        S[k * lds + k] = d;
        f.Dd[k] = d;
        f.Do[k] = 0.0;
        f.pk[k] = 0;
      }
      __syncthreads();
      ++k;
    };
    while (k < pend) {
      const bool mine = tid >= k && tid < m;
      const double v = mine ? column(k, S[k * lds + tid]) : 0.0;
      if (mine) colk[tid] = v;
      if (is_static) {
        __syncthreads();
        double applied;
        const double d = static_pivot(colk[k], sgn[k], floorv, delta, applied);
        if (applied != 0.0) {
          pert += fabs(applied);
          ++nPert;
        }
        finish_1x1(d, v);
        continue;
      }
      ArgMax am = argmax_combine(ArgMax{0.0, -1}, tid > k && tid < effEnd ? ArgMax{fabs(v), tid} : ArgMax{0.0, -1});
      am = warp_argmax_nonneg(am);
      if (lane == 0) {
        arg_v[warp] = am.v;
        arg_i[warp] = am.i;
      }
      __syncthreads();
      am = ArgMax{arg_v[0], arg_i[0]};
#pragma unroll
      for (int w = 1; w < NW; ++w) am = argmax_combine(am, ArgMax{arg_v[w], arg_i[w]});
      const double lambda = am.v, akk = colk[k];
      const int r = am.i;
      int dec;  // 0: 1x1 at k, 1: interchange k <-> r, 1x1, 2: 2x2 (k, r), 3: stop
      double arr = 0.0, vkr = 0.0, u = 0.0;
      if (lambda <= o.zero_tol) {
        const double isolatedFloor = fmax(o.zero_tol, o.rel_floor * orig_max);
        dec = (fabs(akk) <= isolatedFloor) ? 3 : 0;
      } else if (r < 0 || fabs(akk) >= kAlphaBK * lambda) {  // (r < 0: no candidate, under a negative zero_tol)
        dec = 0;
      } else {
        u = mine ? column(r, tid >= r ? S[r * lds + tid] : S[tid * lds + r]) : 0.0;
        if (mine) colr[tid] = u;
        const double smax = warp_max_nonneg(mine && tid < effEnd && tid != r ? fabs(u) : 0.0);
        if (lane == 0) max_v[warp] = smax;
        __syncthreads();
        double sigma = max_v[0];
#pragma unroll
        for (int w = 1; w < NW; ++w) sigma = fmax(sigma, max_v[w]);
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
      if (dec == 0) {
        finish_1x1(akk, v);
        continue;
      }
      if (dec == 1) {
        // the new column k is column r with rows k and r exchanged
        if (tid == r) u = colr[k];
        interchange(k, r);
        finish_1x1(arr, u);
        continue;
      }
      // 2x2: bring r to k + 1
      const double d11 = akk, d21 = vkr, d22 = arr;
      const double det = d11 * d22 - d21 * d21;
      rmax = warp_max_nonneg(rmax);
      if (lane == 0) rm_v[warp] = rmax;
      double a0 = v, a1 = u;
      if (r != k + 1) {
        if (tid == r) {
          a0 = colk[k + 1];
          a1 = colr[k + 1];
        }
        interchange(k + 1, r);
      } else {
        __syncthreads();
      }
      double rm = orig_max;
#pragma unroll
      for (int w = 0; w < NW; ++w) rm = fmax(rm, rm_v[w]);
      const double rm1 = fmax(1.0, rm);
      if (fabs(det) <= o.zero_tol * rm1 * rm1) {
        stopped = true;
        break;
      }
      rmax = fmax(rmax, fmax(fabs(d11), fmax(fabs(d21), fabs(d22))));
      if (det < 0) {
        ++n_pos;
        ++n_neg;
      } else {
        const double tr = d11 + d22;
        if (tr > 0)
          n_pos += 2;
        else if (tr < 0)
          n_neg += 2;
        else {
          ++n_pos;
          ++n_neg;
        }
      }
      const double inv11 = d22 / det, inv21 = -d21 / det, inv22 = d11 / det;
      if (tid >= k + 2 && tid < m) {
        rmax = fmax(rmax, fmax(fabs(a0), fabs(a1)));
        S[k * lds + tid] = a0 * inv11 + a1 * inv21;
        S[(k + 1) * lds + tid] = a0 * inv21 + a1 * inv22;
        W[(k - ks) * kWS + tid] = a0;
        W[(k + 1 - ks) * kWS + tid] = a1;
      } else if (tid == k) {
        S[k * lds + k] = d11;
        S[k * lds + k + 1] = d21;
        S[(k + 1) * lds + k + 1] = d22;
        f.Dd[k] = d11;
        f.Dd[k + 1] = d22;
        f.Do[k] = d21;
        f.Do[k + 1] = 0.0;
        f.pk[k] = 1;
        f.pk[k + 1] = 2;
      }
      __syncthreads();
      k += 2;
    }
    // ---- the rest of the front: S(i, j) -= sum_q L(i, q) W(q, j), i >= j >= k,
    // in 16 x 8 tiles of the lower triangle, the warps in turn
    const int np = k - ks;
    if (np > 0 && k < m) {
      const int rest = m - k, rt_n = (rest + 15) / 16;
      const int gr = lane >> 2, t4 = lane & 3;
      int n = 0;
      for (int rt = 0; rt < rt_n; ++rt) {
        const int i0 = k + 16 * rt;
        for (int j0 = k; j0 <= min(i0 + 15, m - 1); j0 += 8, ++n) {
          if ((n & (NW - 1)) != warp) continue;
          double acc[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int i = i0 + gr + 8 * (e >> 1), j = j0 + 2 * t4 + (e & 1);
            acc[e] = (i < m && j <= i) ? S[j * lds + i] : 0.0;
          }
          for (int q0 = 0; q0 < np; q0 += 8) {
            double a[4], b[2];
#pragma unroll
            for (int x = 0; x < 4; ++x) {
              const int q = q0 + t4 + 4 * (x >> 1), i = i0 + gr + 8 * (x & 1);
              a[x] = (q < np && i < m) ? S[(ks + q) * lds + i] : 0.0;
            }
#pragma unroll
            for (int x = 0; x < 2; ++x) {
              const int q = q0 + t4 + 4 * x, j = j0 + gr;
              b[x] = (q < np && j < m) ? -W[q * kWS + j] : 0.0;
            }
            small_dmma(acc, a, b);
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int i = i0 + gr + 8 * (e >> 1), j = j0 + 2 * t4 + (e & 1);
            if (i < m && j <= i) {
              S[j * lds + i] = acc[e];
              rmax = fmax(rmax, fabs(acc[e]));
            }
          }
        }
      }
      __syncthreads();
    }
  }

  // ---- write back (lower triangle of the whole front, permuted indices)
  for (int j0 = 0; j0 < m; j0 += 8) {
    double v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = (tid < m && j0 + q <= tid) ? S[(j0 + q) * lds + tid] : 0.0;
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (tid < m && j0 + q <= tid) f.F[static_cast<int64_t>(j0 + q) * f.ld + tid] = v[q];
  }
  if (tid < m) {
    f.fidx[tid] = fi[tid];
    f.lperm[tid] = lp[tid];
    f.lpos[lp[tid]] = tid;
  }
  rmax = warp_max_nonneg(rmax);
  __syncthreads();
  if (lane == 0) rm_v[warp] = rmax;
  __syncthreads();
  if (tid == 0) {
    rmax = orig_max;
    for (int w = 0; w < NW; ++w) rmax = fmax(rmax, rm_v[w]);
    FrontState& R = st[s];
    R.npiv = k;
    R.n_pos = n_pos;
    R.n_neg = n_neg;
    R.n_zero = n_zero;
    R.num_perturbed = nPert;
    R.perturb = pert;
    R.orig_max = orig_max;
    R.running_max = rmax;
    R.delta = delta;
    R.k = k;
    int flags = kFlagDone;
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
    R.flags = flags;
  }
}

size_t small_front_smem(int m) {
  return (static_cast<size_t>(front_lds(m)) * m + (kNB + 1) * kWS) * sizeof(double);
}

cudaError_t configure_small_front() {
  return cudaFuncSetAttribute(small_front_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              static_cast<int>(small_front_smem(kSmallFrontMax)));
}

void launch_small_front(const FrontDesc* fronts, const ChildLink* links, FrontState* st, const int* list, int count,
                        int max_m, const int* a_colptr, const KernelOpts& o, FactorGlobals* g, int level, int dynamic,
                        cudaStream_t stream) {
  if (count <= 0) return;
  small_front_kernel<<<count, kNT, small_front_smem(max_m), stream>>>(fronts, links, st, list, a_colptr, o, g, level,
                                                                      dynamic);
}

}  // namespace symla_gpu
