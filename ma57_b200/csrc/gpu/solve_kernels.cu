// Supernodal multi-RHS solve kernels (forward, block-diagonal D^{-1},
// backward) walking the tree level by level, plus the FP64 residual used by
// iterative refinement. sm_100a.
//
// Reference behaviour followed (include/symla/...):
//   solve.hpp:303-362  forward: each front gathers its children's forwarded
//                      deltas (RhsElement), solves with its unit-lower Ltop
//                      (d21 slots of 2x2 blocks masked) and forwards
//                      L_bottom * y for its remaining rows to the parent
//   solve.hpp:434-455  D^{-1} with closed-form 2x2 blocks
//   solve.hpp:364-383  backward: gather ancestor values, subtract
//                      L_bottom^T x, transposed unit-lower solve
//   refine.hpp:116     R = B - A.selfadjointView<Lower>() * X
//
// Work decomposition: every front is cut into 64-row blocks (forward) or
// 64-column blocks of its pivot range (backward); fronts of at most 32 rows
// are taken whole by one warp, eight to a task. One cooperative launch runs
// the tasks of all tree levels, for up to four groups of 16 right-hand sides
// side by side. A block that needs the solution of an earlier block of the
// same front waits for that block's flag (release/acquire), so the triangular
// solve of a large front is pipelined across many SMs instead of running in
// one CTA; a front waits for its children (forward) or its nearest ancestor
// with pivots (backward) on a counter that their tasks raise. Each CTA walks
// its tasks in increasing order and a task only waits on tasks with a smaller
// index, and the launch is cooperative (all CTAs resident), so the waits
// always end; every wait is still bounded and reports a timeout through the
// error word instead of spinning forever.
//
// What bounds it: the chain of a top front's blocks (flag, right-hand sides
// from L2, one tile product, the diagonal block's substitution, store, flag),
// and below the top the latency of a task's dependent loads. A launch
// per level, one warp's worth of work per 256-thread CTA for tiny fronts, the
// groups one after another and scalar tile products took 1.93 ms for one
// right-hand side on a 40^3 27-point grid and 10.6 ms for 37 on 48^3; now 1.23
// and 4.7 ms. A top front's block takes 7.2 us of its chain with 16
// right-hand sides, 9.6 before.
//
// Sign convention: a front's workspace rows for its own pivots hold y after
// the forward pass; its remaining rows hold the negated forwarded delta
// (sum of the children's minus L_bottom * y), so the parent adds them.
#include <cmath>

#include <algorithm>

#include "common.cuh"
#include "factor_kernels.h"
#include "reduce.cuh"

namespace symla_gpu {

namespace {
constexpr int kRB = 64;        // rows (forward) / columns (backward) per block
constexpr int kST = 256;       // threads per CTA
constexpr int kRhsChunk = 16;  // right-hand sides per pass

__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// Wait until *p >= target; false once wait_ns of the global timer or
// wait_ns / 32 unsuccessful probes have passed (the timeout is recorded in
// the error word), or another CTA raised an error. One thread.
__device__ __forceinline__ bool wait_ge(const int* p, int target, int* err, unsigned long long wait_ns) {
  if (ld_acquire(p) >= target) return true;
  const unsigned long long t0 = global_ns();
  const unsigned long long max_probes = wait_ns / 32;
  for (unsigned long long it = 1; ld_acquire(p) < target; ++it) {
    if ((it & 15) == 0 && ld_acquire(err) != 0) return false;
    if (it > max_probes || global_ns() - t0 > wait_ns) {
      atomicCAS(err, 0, kSolveErrTimeout);
      return false;
    }
    __nanosleep(32);
  }
  return true;
}

// The same for the whole CTA (a block barrier).
__device__ __forceinline__ bool cta_wait_ge(const int* p, int target, int* err, unsigned long long wait_ns) {
  const bool ok = threadIdx.x != 0 || wait_ge(p, target, err, wait_ns);
  return !__syncthreads_or(!ok);
}

// After the CTA's stores: raise flag (if any) to epoch and add one to the
// counter (if any).
__device__ __forceinline__ void publish(int* flag, int epoch, int* counter) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (flag) st_release(flag, epoch);
    if (counter) atomicAdd(counter, 1);
  }
}
}  // namespace

__global__ void permute_in_kernel(int n, int nrhs, const int* __restrict__ perm, const double* __restrict__ B, int ldb,
                                  double* __restrict__ Bp, CheckWord* chk) {
  const long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (t >= static_cast<long long>(n) * nrhs) return;
  const int i = static_cast<int>(t % n), c = static_cast<int>(t / n);
  const int p = perm[i];
  Bp[t] = check(in_range(p, 0, n), chk, kChkPermute, i) ? B[p + static_cast<long long>(c) * ldb] : 0.0;
}

__global__ void permute_out_kernel(int n, int nrhs, const int* __restrict__ perm, const double* __restrict__ X,
                                   double* __restrict__ Xout, int ldx, CheckWord* chk) {
  const long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (t >= static_cast<long long>(n) * nrhs) return;
  const int i = static_cast<int>(t % n), c = static_cast<int>(t / n);
  const int p = perm[i];
  if (check(in_range(p, 0, n), chk, kChkPermute, i)) Xout[p + static_cast<long long>(c) * ldx] = X[t];
}

// Checked build: a row index or a child workspace row out of range raises
// the solve's error word (the other CTAs then stop waiting) and the access
// is skipped. The ordinary build compiles this to true.
__device__ __forceinline__ bool solve_index_ok(bool ok, int* err) {
  if constexpr (kCheckedBuild) {
    if (!ok) atomicCAS(err, 0, kSolveErrBounds);
    return ok;
  }
  return true;
}

// Shared-memory layout of both pipelined kernels (dynamic, doubles):
//   T  [2][64][68]  double-buffered L tiles, column-major as the front stores
//                   them (a column's 64 rows consecutive: 16-byte copies, and
//                   a stride that keeps the fragment loads of both products
//                   conflict-free); the backward diagonal block is read along
//                   rows and takes a stride of 65 instead
//   xb [64][20]     the right-hand-side block of the current tile
//   acc[64][20]     the task's result block
// Every L tile a task needs is known from its position alone, so the next
// tile is copied (cp.async) while the current one is used and before the
// flag that guards its right-hand side is awaited.
constexpr int kTS = 68;
constexpr int kTSDiag = 65;
constexpr int kXS = 20;
constexpr size_t kSolveSmem = (2 * kRB * kTS + 2 * kRB * kXS) * sizeof(double);
constexpr int kTinyRows = 32;  // fronts of at most this many rows: one warp each

template <int Bytes>
__device__ __forceinline__ void scp_async(double* smem_dst, const double* gsrc) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(d), "l"(gsrc), "n"(Bytes) : "memory");
}
__device__ __forceinline__ void scp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void scp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// Tile (rows [i0, i0 + ni), columns [j0, j0 + nj)) of a front into T,
// T[jj * kTS + ii]; entries outside the ranges are zero. i0 is even and the
// front's columns start on 16-byte boundaries.
__device__ __forceinline__ void stage_tile(double* T, const double* F, int64_t ld, int i0, int ni, int j0, int nj) {
  for (int t = threadIdx.x; t < kRB * kRB / 2; t += kST) {
    const int ii = 2 * (t % (kRB / 2)), jj = t / (kRB / 2);
    double* d = T + jj * kTS + ii;
    const double* src = F + static_cast<int64_t>(j0 + jj) * ld + i0 + ii;
    if (ii + 1 < ni && jj < nj) {
      scp_async<16>(d, src);
    } else {
      d[1] = 0.0;
      if (ii < ni && jj < nj)
        scp_async<8>(d, src);
      else
        d[0] = 0.0;
    }
  }
  scp_commit();
}
// An n x n diagonal block at (q0, q0) into T[jj * kTSDiag + ii].
__device__ __forceinline__ void stage_diag(double* T, const double* F, int64_t ld, int q0, int n) {
  for (int t = threadIdx.x; t < kRB * kRB; t += kST) {
    const int ii = t % kRB, jj = t / kRB;
    if (ii < n && jj < n) scp_async<8>(T + jj * kTSDiag + ii, F + static_cast<int64_t>(q0 + jj) * ld + q0 + ii);
  }
  scp_commit();
}

// c (16 x 8) += a (16 x 8) * b (8 x 8) on the FP64 tensor path; fragments as in
// update_mma_kernel
__device__ __forceinline__ void solve_dmma(double* c, const double* a, const double* b) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
               : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

// The 64 x 64 by 64 x 16 product of a tile, summed over a block's tiles in
// registers: warp w takes rows 16 (w & 3) and, of the right-hand sides, the
// eight from 8 (w >> 2); with at most eight of them, warps 4 .. 7 take the
// second half of the tile's inner dimension of the same eight instead.
// Trans: the product with the tile's transpose (backward).
template <bool Trans>
struct TileProduct {
  double sum[4] = {0.0, 0.0, 0.0, 0.0};
  __device__ __forceinline__ void add(const double* T, const double* xb, int nc) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int r0 = 16 * (warp & 3), hi = warp >> 2;
    const bool split = nc <= 8;
    const int k0 = split ? 32 * hi : 0, c0 = split ? 0 : 8 * hi;
    const int ksteps = split ? 4 : 8;
    // each tile's products are summed apart: one chain over thousands of rows
    // loses two to three times as much (measured on 48^3 solves)
    double p[2][4] = {};
#pragma unroll 4
    for (int ks = 0; ks < ksteps; ++ks) {
      const int k = k0 + 8 * ks;
      double a[4], b[2];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int row = r0 + g + 8 * (r & 1), kk = k + t + 4 * (r >> 1);
        a[r] = Trans ? T[row * kTS + kk] : T[kk * kTS + row];
      }
#pragma unroll
      for (int r = 0; r < 2; ++r) b[r] = xb[(k + t + 4 * r) * kXS + c0 + g];
      solve_dmma(p[ks & 1], a, b);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) sum[e] += p[0][e] + p[1][e];
  }
  // acc[row][c] -= the product for row < rows, c < nc (a block barrier inside
  // when the inner dimension was split)
  __device__ __forceinline__ void subtract_into(double* acc, int rows, int nc) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int r0 = 16 * (warp & 3), hi = warp >> 2;
    const bool split = nc <= 8;
    const int c0 = split ? 0 : 8 * hi;
    auto put = [&] {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int row = r0 + g + 8 * (e >> 1), c = c0 + 2 * t + (e & 1);
        if (row < rows && c < nc) acc[row * kXS + c] -= sum[e];
      }
    };
    if (!split || hi == 0) put();
    if (split) {
      __syncthreads();
      if (hi == 1) put();
    }
  }
};

// ---------------------------------------------------------------------------
// Forward: one front of at most 32 rows by one warp, lane = row.
__device__ bool forward_tiny(const FrontDesc* __restrict__ fronts, const ChildLink* __restrict__ links,
                             const FrontState* __restrict__ st, int s, const SolvePlan& pl, int* counters, int* err,
                             unsigned long long wait_ns, int nc, int c0, const double* __restrict__ Bp, int n) {
  const int lane = threadIdx.x & 31;
  const FrontDesc f = fronts[s];
  const int m = f.m, np = st[s].npiv;
  const int64_t ld = f.ld;
  double y[kRhsChunk];
#pragma unroll
  for (int c = 0; c < kRhsChunk; ++c) y[c] = 0.0;
  const int gi = lane < np ? f.fidx[lane] : 0;
  if (lane < np && solve_index_ok(in_range(gi, 0, n), err))
#pragma unroll
    for (int c = 0; c < kRhsChunk; ++c)
      if (c < nc) y[c] = Bp[gi + static_cast<int64_t>(c0 + c) * n];
  const int need = pl.fwd_need[s];
  if (need > 0) {
    const bool ok = lane != 0 || wait_ge(counters + s, need, err, wait_ns);
    if (!__all_sync(0xffffffffu, ok)) return false;
    __syncwarp();
    if (lane < m) {
      const int pre = f.lperm[lane];
      for (int ch = f.ch_begin; ch < f.ch_end; ++ch) {
        const ChildLink L = links[ch];
        const int a = L.invmap[pre];
        if (a < 0) continue;
        const FrontDesc& cf = fronts[L.child];
        const int cnp = st[L.child].npiv;
        if (solve_index_ok(cnp >= 0 && cnp + a < cf.m, err)) {
          const double* w = cf.W + cnp + a + static_cast<int64_t>(c0) * cf.wld;
#pragma unroll
          for (int c = 0; c < kRhsChunk; ++c)
            if (c < nc) y[c] += w[static_cast<int64_t>(c) * cf.wld];
        }
      }
    }
    __syncwarp();
  }
  for (int j0 = 0; j0 < np; j0 += 4) {
    double l[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int j = j0 + q;
      // (the slot below a 2x2 pivot's first column holds d21, not L)
      l[q] = (j < np && lane > j && lane < m && !(f.pk[j] == 1 && lane == j + 1)) ? f.F[j * ld + lane] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (j0 + q < np)
#pragma unroll
        for (int c = 0; c < kRhsChunk; ++c)
          if (c < nc) y[c] = fma(-l[q], __shfl_sync(0xffffffffu, y[c], j0 + q), y[c]);
  }
  if (lane < m) {
    double* w = f.W + lane + static_cast<int64_t>(c0) * f.wld;
#pragma unroll
    for (int c = 0; c < kRhsChunk; ++c)
      if (c < nc) w[static_cast<int64_t>(c) * f.wld] = y[c];
  }
  __syncwarp();
  if (lane == 0 && f.parent >= 0) {
    __threadfence();
    atomicAdd(counters + f.parent, 1);
  }
  return true;
}

// Forward: one row block (front s, block rb). Returns false when a wait
// ended in an error (the CTA then leaves the launch).
__device__ bool forward_block(const FrontDesc* __restrict__ fronts, const ChildLink* __restrict__ links,
                              const FrontState* __restrict__ st, int s, int rb, const SolvePlan& pl, int* flags,
                              int* counters, int epoch, int* err, unsigned long long wait_ns, int nc, int c0,
                              const double* __restrict__ Bp, int n, double* acc, double* xb, double* Lb0) {
  const FrontDesc f = fronts[s];
  const int m = f.m, np = st[s].npiv;
  const int r0 = rb * kRB, r1 = min(r0 + kRB, m), nr = r1 - r0;
  const int64_t ld = f.ld;
  double* W = f.W;
  const int wld = f.wld;
  const int nbp = (np + kRB - 1) / kRB;
  const int jend = min(rb, nbp);
  const bool hasDiag = r0 < np;
  const int ntiles = jend + (hasDiag ? 1 : 0);
  const int fbase = pl.flag_base[s];
  // pivot kinds the steps below need, loaded before any wait: a 2x2 pivot
  // ending at row r0 - 1 (its d21 slot sits in the last earlier tile) and
  // one starting at this thread's row of the diagonal block
  const bool pair_before = r0 > 0 && r0 - 1 < np && f.pk[r0 - 1] == 1;
  const bool own_pair = hasDiag && threadIdx.x + 1 < min(r1, np) - r0 && f.pk[r0 + threadIdx.x] == 1;
  // tile tt: pivot block tt (tt < jend) or the diagonal block
  auto stage = [&](int tt) {
    double* T = Lb0 + (tt & 1) * kRB * kTS;
    if (tt < jend) {
      const int j0 = tt * kRB;
      stage_tile(T, f.F, ld, r0, nr, j0, min(j0 + kRB, np) - j0);
    } else {
      stage_tile(T, f.F, ld, r0, nr, r0, min(r1, np) - r0);
    }
  };
  if (ntiles > 0) stage(0);
  // 1. Bp for pivot rows plus the children's forwarded rows, gathered
  //    through each row's pre-pivot position
  const int need = pl.fwd_need[s];
  if (need > 0 && !cta_wait_ge(counters + s, need, err, wait_ns)) {
    scp_wait<0>();
    return false;
  }
  for (int t = threadIdx.x; t < nr * nc; t += kST) {
    const int ii = t % nr, c = t / nr;
    const int i = r0 + ii;
    double v = 0.0;
    if (i < np) {
      const int gi = f.fidx[i];
      if (solve_index_ok(in_range(gi, 0, n), err)) v = Bp[gi + static_cast<int64_t>(c0 + c) * n];
    }
    const int pre = f.lperm[i];
    for (int ch = f.ch_begin; ch < f.ch_end; ++ch) {
      const ChildLink L = links[ch];
      const int a = L.invmap[pre];
      if (a < 0) continue;
      const FrontDesc& cf = fronts[L.child];
      const int cnp = st[L.child].npiv;
      if (solve_index_ok(cnp >= 0 && cnp + a < cf.m, err)) v += cf.W[cnp + a + static_cast<int64_t>(c0 + c) * cf.wld];
    }
    acc[ii * kXS + c] = v;
  }
  TileProduct<false> prod;
  for (int tt = 0; tt < jend; ++tt) {
    // 2. contribution of finished pivot block tt
    const bool more = tt + 1 < ntiles;
    if (more) stage(tt + 1);
    double* T = Lb0 + (tt & 1) * kRB * kTS;
    if (!cta_wait_ge(flags + fbase + tt, epoch, err, wait_ns)) {
      scp_wait<0>();
      return false;
    }
    const int j0 = tt * kRB, nj = min(j0 + kRB, np) - j0;
    for (int t = threadIdx.x; t < kRB * kRhsChunk; t += kST) {
      const int jj = t % kRB, c = t / kRB;
      xb[jj * kXS + c] = (jj < nj && c < nc) ? W[j0 + jj + static_cast<int64_t>(c0 + c) * wld] : 0.0;
    }
    if (more)
      scp_wait<1>();
    else
      scp_wait<0>();
    __syncthreads();
    // a 2x2 pivot straddling the block boundary: its d21 slot in L is not
    // an L entry
    if (pair_before && tt == rb - 1) {
      if (threadIdx.x == 0) T[(r0 - 1 - j0) * kTS] = 0.0;
      __syncthreads();
    }
    prod.add(T, xb, nc);
    __syncthreads();
  }
  if (jend > 0) prod.subtract_into(acc, nr, nc);
  if (hasDiag) {
    // 3. the block's own pivot columns: unit-lower solve for its pivot
    //    rows and the matching update of its non-pivot rows
    double* T = Lb0 + (jend & 1) * kRB * kTS;
    scp_wait<0>();
    __syncthreads();
    const int npv = min(r1, np) - r0;
    if (own_pair) T[threadIdx.x * kTS + threadIdx.x + 1] = 0.0;  // d21 slot of a 2x2 pivot
    __syncthreads();
    // a warp takes right-hand sides c and c + 8 together: the two
    // substitution chains interleave (each step is a shuffle and an FMA)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int NW = kST / 32;
    for (int c = warp; c < nc; c += 2 * NW) {
      const int cb = c + NW;
      const bool two = cb < nc;
      double y0 = (lane < nr) ? acc[lane * kXS + c] : 0.0;
      double y1 = (lane + 32 < nr) ? acc[(lane + 32) * kXS + c] : 0.0;
      double z0 = (two && lane < nr) ? acc[lane * kXS + cb] : 0.0;
      double z1 = (two && lane + 32 < nr) ? acc[(lane + 32) * kXS + cb] : 0.0;
      const int nlow = min(npv, 32);
#pragma unroll 8
      for (int jj = 0; jj < nlow; ++jj) {
        const double yj = __shfl_sync(0xffffffffu, y0, jj), zj = __shfl_sync(0xffffffffu, z0, jj);
        const double t0 = T[jj * kTS + lane], t1 = T[jj * kTS + lane + 32];
        if (lane > jj) {
          y0 -= t0 * yj;
          z0 -= t0 * zj;
        }
        y1 -= t1 * yj;
        z1 -= t1 * zj;
      }
#pragma unroll 8
      for (int jj = 32; jj < npv; ++jj) {
        const double yj = __shfl_sync(0xffffffffu, y1, jj - 32), zj = __shfl_sync(0xffffffffu, z1, jj - 32);
        const double t1 = T[jj * kTS + lane + 32];
        if (lane + 32 > jj) {
          y1 -= t1 * yj;
          z1 -= t1 * zj;
        }
      }
      if (lane < nr) acc[lane * kXS + c] = y0;
      if (lane + 32 < nr) acc[(lane + 32) * kXS + c] = y1;
      if (two && lane < nr) acc[lane * kXS + cb] = z0;
      if (two && lane + 32 < nr) acc[(lane + 32) * kXS + cb] = z1;
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < nr * nc; t += kST) {
    const int ii = t % nr, c = t / nr;
    W[r0 + ii + static_cast<int64_t>(c0 + c) * wld] = acc[ii * kXS + c];
  }
  publish(hasDiag ? flags + fbase + rb : nullptr, epoch, f.parent >= 0 ? counters + f.parent : nullptr);
  __syncthreads();
  return true;
}

// Forward task = int4 {front, row block, 0, 0} or {first, -2, count, 0}: the
// fronts pl.tiny[first ..], a warp each. Flag of a pivot row block at
// flag_base[front] + row block. Task t of the launch is task t / nchunks of
// the list for right-hand-side group t % nchunks (16 from c0 + 16 of it),
// whose flags and counters are its own.
__global__ void __launch_bounds__(kST, 2) forward_pipelined_kernel(
    const FrontDesc* __restrict__ fronts, const ChildLink* __restrict__ links, const FrontState* __restrict__ st,
    SolvePlan pl, int task0, int ntasks, int nchunks, int epoch, int* err, unsigned long long wait_ns, int nrhs, int c0,
    const double* __restrict__ Bp, int n) {
  extern __shared__ __align__(16) double ssm[];
  double* Lb0 = ssm;
  double* xb = Lb0 + 2 * kRB * kTS;
  double* acc = xb + kRB * kXS;
  for (int t = blockIdx.x; t < ntasks * nchunks; t += gridDim.x) {
    if (ld_acquire(err) != 0) return;
    const int chunk = t % nchunks, cc0 = c0 + chunk * kRhsChunk, nc = min(kRhsChunk, nrhs - cc0);
    const int4 tk = pl.fwd_tasks[task0 + t / nchunks];
    int* flags = pl.flags + static_cast<int64_t>(chunk) * pl.nflags;
    int* counters = pl.counters + static_cast<int64_t>(chunk) * pl.nfronts;
    if (tk.y >= 0) {
      if (!forward_block(fronts, links, st, tk.x, tk.y, pl, flags, counters, epoch, err, wait_ns, nc, cc0, Bp, n, acc,
                         xb, Lb0))
        return;
    } else {
      const int w = threadIdx.x >> 5;
      const bool ok = w >= tk.z || forward_tiny(fronts, links, st, pl.tiny[tk.x + w], pl, counters, err, wait_ns, nc,
                                                cc0, Bp, n);
      if (__syncthreads_or(!ok)) return;
    }
  }
}

// ---------------------------------------------------------------------------
// z = (D^{-1} y)_q of a front's pivot q (w: a right-hand side's column of W)
__device__ __forceinline__ double d_inverse(const FrontDesc& f, const double* w, int q) {
  const int8_t kind = f.pk[q];
  if (kind == 0) return w[q] / f.Dd[q];
  const int a = kind == 1 ? q : q - 1;
  const double d11 = f.Dd[a], d21 = f.Do[a], d22 = f.Dd[a + 1];
  const double det = d11 * d22 - d21 * d21;
  return (kind == 1 ? d22 * w[q] - d21 * w[q + 1] : -d21 * w[q - 1] + d11 * w[q]) / det;
}

// Backward: one front of at most 32 rows by one warp; lanes below npiv hold
// its unknowns, the others its ancestors' values.
__device__ bool backward_tiny(const FrontDesc* __restrict__ fronts, const FrontState* __restrict__ st, int s,
                              const SolvePlan& pl, int* counters, int* err, unsigned long long wait_ns, int nc, int c0,
                              double* __restrict__ X, int n) {
  const int lane = threadIdx.x & 31;
  const FrontDesc f = fronts[s];
  const int m = f.m, np = st[s].npiv;
  const int64_t ld = f.ld;
  double x[kRhsChunk];
#pragma unroll
  for (int c = 0; c < kRhsChunk; ++c)
    x[c] = (lane < np && c < nc) ? d_inverse(f, f.W + static_cast<int64_t>(c0 + c) * f.wld, lane) : 0.0;
  const int gi = lane < m ? f.fidx[lane] : 0;
  const bool idx_ok = lane < m && solve_index_ok(in_range(gi, 0, n), err);
  const bool pair = lane < np && f.pk[lane] == 1;
  const int anc = pl.bwd_wait[s];
  if (anc >= 0) {
    const bool ok = lane != 0 || wait_ge(counters + anc, pl.bwd_need[s], err, wait_ns);
    if (!__all_sync(0xffffffffu, ok)) return false;
    __syncwarp();
    if (lane >= np && idx_ok)
#pragma unroll
      for (int c = 0; c < kRhsChunk; ++c)
        if (c < nc) x[c] = X[gi + static_cast<int64_t>(c0 + c) * n];
  }
  // row r's value is final once every row below it has been applied
  for (int r0 = m - 1; r0 > 0; r0 -= 4) {
    double l[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = r0 - q;
      l[q] = (r > lane && lane < np && !(pair && r == lane + 1)) ? f.F[lane * ld + r] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (r0 - q > 0)
#pragma unroll
        for (int c = 0; c < kRhsChunk; ++c)
          if (c < nc) x[c] = fma(-l[q], __shfl_sync(0xffffffffu, x[c], r0 - q), x[c]);
  }
  if (lane < np && idx_ok)
#pragma unroll
    for (int c = 0; c < kRhsChunk; ++c)
      if (c < nc) X[gi + static_cast<int64_t>(c0 + c) * n] = x[c];
  __syncwarp();
  if (lane == 0 && np > 0) {
    __threadfence();
    atomicAdd(counters + s, 1);
  }
  return true;
}

// Backward: pivot column block cb of front s. The tiles are the ancestor
// rows [np, m) in 64-row chunks, then the later pivot blocks, then the
// diagonal block. A main part (part 0) does ancestor chunks [a0, a1), the
// later blocks, adds its helper parts' partial sums (slots hslot0 ..
// hslot0 + nh - 1, in slot order) and finishes the block; a helper part
// only sums its ancestor chunks into its scratch slot and raises its flag.
// (np need not be a multiple of 64: an ancestor chunk starts at an even row,
// at or one before its first, so that its columns stay 16-byte aligned.)
__device__ bool backward_block(const FrontDesc* __restrict__ fronts, const FrontState* __restrict__ st, int s, int cb,
                               bool helper, int a0, int a1, int hslot0, int nh, const SolvePlan& pl, int* flags,
                               int* hflags, double* hscratch, int* counters, int epoch, int* err,
                               unsigned long long wait_ns, int nc, int c0, double* __restrict__ X, int n, double* acc,
                               double* xb, double* Lb0) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int NW = kST / 32;
  const FrontDesc f = fronts[s];
  const int m = f.m, np = st[s].npiv;
  const int q0 = cb * kRB, q1 = min(q0 + kRB, np), nq = q1 - q0;
  const int64_t ld = f.ld;
  const double* W = f.W;
  const int wld = f.wld;
  const int nbp = (np + kRB - 1) / kRB;
  const int nanc = a1 - a0;
  const int nlater = helper ? 0 : nbp - 1 - cb;
  const int ntiles = nanc + nlater + (helper ? 0 : 1);
  const int fbase = pl.flag_base[s];
  // loaded before any wait: the 2x2 pivot kinds the steps below need and
  // the rows the block's solution is written to
  static_assert(kST % kRB == 0, "a thread keeps one tile row in the gathers");
  __shared__ int s_row[kRB];
  const bool pair_at_end = nq > 0 && f.pk[q1 - 1] == 1;
  const bool own_pair = threadIdx.x + 1 < nq && f.pk[q0 + threadIdx.x] == 1;
  if (!helper && threadIdx.x < nq) s_row[threadIdx.x] = f.fidx[q0 + threadIdx.x];
  const int anc0 = np & ~1;  // ancestor chunks: rows [anc0 + 64 a, ...) without those below np
  auto tile_rows = [&](int tt, int& i0, int& i1) {
    if (tt < nanc) {
      i0 = anc0 + (a0 + tt) * kRB;
      i1 = min(i0 + kRB, m);
    } else {
      const int j = nbp - 1 - (tt - nanc);
      i0 = j * kRB;
      i1 = min(i0 + kRB, np);
    }
  };
  auto stage = [&](int tt) {
    double* T = Lb0 + (tt & 1) * kRB * kTS;
    if (tt < nanc + nlater) {
      int i0, i1;
      tile_rows(tt, i0, i1);
      stage_tile(T, f.F, ld, i0, i1 - i0, q0, nq);
    } else {
      stage_diag(T, f.F, ld, q0, nq);
    }
  };
  if (ntiles > 0) stage(0);
  if (helper) {
    for (int t = threadIdx.x; t < kRB * nc; t += kST) acc[(t % kRB) * kXS + t / kRB] = 0.0;
  } else {
    // 1. z = D^{-1} y for the block's pivots (a 2x2 partner may sit in the
    //    neighbouring block; y is complete in W after the forward pass)
    for (int t = threadIdx.x; t < nq * nc; t += kST) {
      const int qq = t % nq, c = t / nq;
      acc[qq * kXS + c] = d_inverse(f, W + static_cast<int64_t>(c0 + c) * wld, q0 + qq);
    }
  }
  // the ancestors' values are complete once the nearest ancestor with pivots is
  const int anc = nanc > 0 ? pl.bwd_wait[s] : -1;
  if (anc >= 0 && !cta_wait_ge(counters + anc, pl.bwd_need[s], err, wait_ns)) {
    scp_wait<0>();
    return false;
  }
  TileProduct<true> prod;
  for (int tt = 0; tt < nanc + nlater; ++tt) {
    // 2. minus L(rows of the tile, block)^T x(rows of the tile); later pivot
    //    blocks of this front are waited for
    const bool more = tt + 1 < ntiles;
    if (more) stage(tt + 1);
    double* T = Lb0 + (tt & 1) * kRB * kTS;
    int i0, i1;
    tile_rows(tt, i0, i1);
    const int first = tt < nanc ? np : i0;  // rows of the tile before it are not the tile's
    // this thread's tile row (the same for every t below), before the wait
    const int my_i = i0 + static_cast<int>(threadIdx.x) % kRB;
    const bool mine = my_i >= first && my_i < i1;
    const int my_gi = mine ? f.fidx[my_i] : 0;
    if (tt >= nanc) {
      const int j = nbp - 1 - (tt - nanc);
      if (!cta_wait_ge(flags + fbase + j, epoch, err, wait_ns)) {
        scp_wait<0>();
        return false;
      }
    }
    const bool load = mine && solve_index_ok(in_range(my_gi, 0, n), err);
    for (int t = threadIdx.x; t < kRB * kRhsChunk; t += kST) {
      const int c = t / kRB;
      xb[(t % kRB) * kXS + c] = (load && c < nc) ? X[my_gi + static_cast<int64_t>(c0 + c) * n] : 0.0;
    }
    if (more)
      scp_wait<1>();
    else
      scp_wait<0>();
    __syncthreads();
    // a 2x2 pivot straddling the block boundary: its d21 slot (row q1) is not
    // an L entry; the pivot row before an odd np is not the chunk's
    const bool odd_row = first > i0, straddle = pair_at_end && i0 == q1;
    if (odd_row || straddle) {
      if (odd_row && threadIdx.x < kRB) T[threadIdx.x * kTS] = 0.0;
      if (straddle && threadIdx.x == 0) T[(nq - 1) * kTS] = 0.0;
      __syncthreads();
    }
    prod.add(T, xb, nc);
    __syncthreads();
  }
  if (nanc + nlater > 0) prod.subtract_into(acc, nq, nc);
  __syncthreads();
  if (helper) {
    // acc holds minus the helper's partial sum; the main part adds it
    double* part = hscratch + static_cast<int64_t>(hslot0) * kRB * kRhsChunk;
    for (int t = threadIdx.x; t < nq * nc; t += kST) {
      const int qq = t % nq, c = t / nq;
      part[c * kRB + qq] = acc[qq * kXS + c];
    }
    publish(hflags + hslot0, epoch, nullptr);
    __syncthreads();
    return true;
  }
  // helper parts' partial sums, in slot order (deterministic)
  for (int h = 0; h < nh; ++h) {
    if (!cta_wait_ge(hflags + hslot0 + h, epoch, err, wait_ns)) {
      scp_wait<0>();
      return false;
    }
    const double* part = hscratch + static_cast<int64_t>(hslot0 + h) * kRB * kRhsChunk;
    for (int t = threadIdx.x; t < nq * nc; t += kST) {
      const int qq = t % nq, c = t / nq;
      acc[qq * kXS + c] += part[c * kRB + qq];
    }
  }
  // 3. transposed unit-lower solve on the diagonal block
  double* T = Lb0 + ((nanc + nlater) & 1) * kRB * kTS;
  scp_wait<0>();
  __syncthreads();
  if (own_pair) T[threadIdx.x * kTSDiag + threadIdx.x + 1] = 0.0;  // d21 slot of a 2x2 pivot
  __syncthreads();
  // right-hand sides c and c + NW together (interleaved chains)
  for (int c = warp; c < nc; c += 2 * NW) {
    const int cb2 = c + NW;
    const bool two = cb2 < nc;
    double x0 = (lane < nq) ? acc[lane * kXS + c] : 0.0;
    double x1 = (lane + 32 < nq) ? acc[(lane + 32) * kXS + c] : 0.0;
    double u0 = (two && lane < nq) ? acc[lane * kXS + cb2] : 0.0;
    double u1 = (two && lane + 32 < nq) ? acc[(lane + 32) * kXS + cb2] : 0.0;
    // x[jj] is final once every row below it has been applied; row jj of
    // Ltop then updates the unknowns above it
#pragma unroll 8
    for (int jj = nq - 1; jj >= 32; --jj) {
      const double xj = __shfl_sync(0xffffffffu, x1, jj - 32), uj = __shfl_sync(0xffffffffu, u1, jj - 32);
      const double t0 = T[lane * kTSDiag + jj];
      x0 -= t0 * xj;
      u0 -= t0 * uj;
      if (lane + 32 < jj) {
        const double t1 = T[(lane + 32) * kTSDiag + jj];
        x1 -= t1 * xj;
        u1 -= t1 * uj;
      }
    }
#pragma unroll 8
    for (int jj = min(nq, 32) - 1; jj >= 0; --jj) {
      const double xj = __shfl_sync(0xffffffffu, x0, jj), uj = __shfl_sync(0xffffffffu, u0, jj);
      if (lane < jj) {
        const double t0 = T[lane * kTSDiag + jj];
        x0 -= t0 * xj;
        u0 -= t0 * uj;
      }
    }
    if (lane < nq) acc[lane * kXS + c] = x0;
    if (lane + 32 < nq) acc[(lane + 32) * kXS + c] = x1;
    if (two && lane < nq) acc[lane * kXS + cb2] = u0;
    if (two && lane + 32 < nq) acc[(lane + 32) * kXS + cb2] = u1;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < nq * nc; t += kST) {
    const int qq = t % nq, c = t / nq;
    const int gi = s_row[qq];
    if (solve_index_ok(in_range(gi, 0, n), err)) X[gi + static_cast<int64_t>(c0 + c) * n] = acc[qq * kXS + c];
  }
  publish(flags + fbase + cb, epoch, counters + s);
  __syncthreads();
  return true;
}

// Number of 64-row ancestor chunks of a front (from the even row at or
// before np).
__host__ __device__ inline int ancestor_chunks(int m, int np) { return m > np ? (m - (np & ~1) + kRB - 1) / kRB : 0; }

// Backward task = int4 {front, column block, part, aux}:
//   {first, -2, count, 0}     the fronts pl.tiny[first ..], a warp each
//   {s, -1, 0, 0}             the whole front (blocks last to first, this CTA)
//   {s, cb, 0, P << 20 | h0}  main part of block cb with P parts in all; its
//                             helpers hold scratch slots h0 .. h0 + P - 2
//   {s, cb, p, P << 20 | h}   helper part p (1 <= p < P) in slot h
// The ancestor chunks of a block are split evenly over its P parts. Helpers
// are listed before their main part, and later blocks of a front before
// earlier ones, so every wait is on a task with a smaller index. Tasks of the
// launch as in forward_pipelined_kernel.
__global__ void __launch_bounds__(kST, 2) backward_pipelined_kernel(
    const FrontDesc* __restrict__ fronts, const FrontState* __restrict__ st, SolvePlan pl, int task0, int ntasks,
    int nchunks, int epoch, int* err, unsigned long long wait_ns, int nrhs, int c0, double* __restrict__ X, int n) {
  extern __shared__ __align__(16) double ssm[];
  double* Lb0 = ssm;
  double* xb = Lb0 + 2 * kRB * kTS;
  double* acc = xb + kRB * kXS;
  for (int t = blockIdx.x; t < ntasks * nchunks; t += gridDim.x) {
    if (ld_acquire(err) != 0) return;
    const int chunk = t % nchunks, cc0 = c0 + chunk * kRhsChunk, nc = min(kRhsChunk, nrhs - cc0);
    const int4 tk = pl.bwd_tasks[task0 + t / nchunks];
    int* flags = pl.flags + static_cast<int64_t>(chunk) * pl.nflags;
    int* counters = pl.counters + static_cast<int64_t>(chunk) * pl.nfronts;
    int* hflags = pl.hflags + static_cast<int64_t>(chunk) * pl.nslots;
    double* hscratch = pl.hscratch + static_cast<int64_t>(chunk) * pl.nslots * kRB * kRhsChunk;
    if (tk.y == -2) {
      const int w = threadIdx.x >> 5;
      const bool ok = w >= tk.z || backward_tiny(fronts, st, pl.tiny[tk.x + w], pl, counters, err, wait_ns, nc, cc0, X, n);
      if (__syncthreads_or(!ok)) return;
      continue;
    }
    const int s = tk.x;
    const int m = fronts[s].m, np = st[s].npiv;
    const int nanc = ancestor_chunks(m, np);
    if (tk.y < 0) {
      const int nbp = (np + kRB - 1) / kRB;
      for (int cb = nbp - 1; cb >= 0; --cb)
        if (!backward_block(fronts, st, s, cb, false, 0, nanc, 0, 0, pl, flags, hflags, hscratch, counters, epoch, err,
                            wait_ns, nc, cc0, X, n, acc, xb, Lb0))
          return;
    } else {
      const int P = tk.w >> 20, slot = tk.w & ((1 << 20) - 1), p = tk.z;
      const int a0 = static_cast<int>(static_cast<long long>(nanc) * p / P);
      const int a1 = static_cast<int>(static_cast<long long>(nanc) * (p + 1) / P);
      if (!backward_block(fronts, st, s, tk.y, p > 0, a0, a1, slot, p > 0 ? 1 : P - 1, pl, flags, hflags, hscratch,
                          counters, epoch, err, wait_ns, nc, cc0, X, n, acc, xb, Lb0))
        return;
    }
  }
}

__global__ void residual_kernel(int n, int nrhs, const int* __restrict__ rowptr, const int* __restrict__ colind,
                                const int* __restrict__ vidx, const double* __restrict__ vals,
                                const double* __restrict__ X, int ldx, const double* __restrict__ B, int ldb,
                                double* __restrict__ R) {
  const long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (t >= static_cast<long long>(n) * nrhs) return;
  const int i = static_cast<int>(t % n), c = static_cast<int>(t / n);
  const double* x = X + static_cast<long long>(c) * ldx;
  double acc = 0.0;
  for (int e = rowptr[i]; e < rowptr[i + 1]; ++e) acc += vals[vidx[e]] * x[colind[e]];
  R[i + static_cast<long long>(c) * n] = B[i + static_cast<long long>(c) * ldb] - acc;
}

// The norms of the refinement propagate a NaN (the bit-pattern maximum of
// non-negative values orders NaN above +Inf), so a non-finite residual or
// solution can never read as converged.
__global__ void absmax_kernel(const double* __restrict__ v, long long len, double* out) {
  double m = 0.0;
  for (long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; t < len;
       t += static_cast<long long>(gridDim.x) * blockDim.x)
    m = nan_sticky_absmax(m, v[t]);
  m = warp_max_nonneg(m);
  if ((threadIdx.x & 31) == 0) atomic_max_nonneg(out, m);
}

__global__ void rowsum_max_kernel(int n, const int* __restrict__ srowptr, const int* __restrict__ svidx,
                                  const double* __restrict__ vals, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double s = 0.0;
  if (i < n)
    for (int e = srowptr[i]; e < srowptr[i + 1]; ++e) s += fabs(vals[svidx[e]]);
  s = warp_max_nonneg(fabs(s));
  if ((threadIdx.x & 31) == 0) atomic_max_nonneg(out, s);
}

__global__ void axpy_kernel(long long len, const double* __restrict__ dx, double* __restrict__ x) {
  const long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (t < len) x[t] += dx[t];
}

__global__ void copy2d_kernel(int rows, int cols, const double* __restrict__ src, int lds, double* __restrict__ dst,
                              int ldd) {
  const long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (t >= static_cast<long long>(rows) * cols) return;
  const int i = static_cast<int>(t % rows), c = static_cast<int>(t / rows);
  dst[i + static_cast<long long>(c) * ldd] = src[i + static_cast<long long>(c) * lds];
}

// ---------------------------------------------------------------------------
// Column-wise vector kernels of GMRES-IR. The Krylov vectors of all
// right-hand sides advance together: vector i, right-hand side c is
// V + i * vs + c * n (n rows, compact).

// partial[(i * nrhs + c) * G + b] = sum over block b's rows of
// V_i[:, c] . W[:, c], with G = gridDim.x; every block sums its rows in a
// fixed order (the host adds the partials in a fixed order too).
__global__ void multi_dot_kernel(int n, int nrhs, const double* __restrict__ V, long long vs,
                                 const double* __restrict__ W, double* __restrict__ partial) {
  __shared__ double red[8];
  const int c = blockIdx.y, i = blockIdx.z;
  const double* v = V + i * vs + static_cast<long long>(c) * n;
  const double* w = W + static_cast<long long>(c) * n;
  double s = 0.0;
  for (long long r = blockIdx.x * 256LL + threadIdx.x; r < n; r += static_cast<long long>(gridDim.x) * 256)
    s = fma(v[r], w[r], s);
  for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int k = 0; k < 8; ++k) t += red[k];
    partial[(static_cast<long long>(i) * nrhs + c) * gridDim.x + blockIdx.x] = t;
  }
}

// W[:, c] -= sum_i coef[i * nrhs + c] * V_i[:, c]
__global__ void multi_axpy_kernel(int n, int nrhs, int nvec, const double* __restrict__ V, long long vs,
                                  const double* __restrict__ coef, double* __restrict__ W) {
  const long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (t >= static_cast<long long>(n) * nrhs) return;
  const int c = static_cast<int>(t / n);
  double acc = W[t];
  for (int i = 0; i < nvec; ++i) acc -= coef[i * nrhs + c] * V[i * vs + t];
  W[t] = acc;
}

// Y[:, c] = alpha[c] * X[:, c]
__global__ void col_scale_kernel(int n, int nrhs, const double* __restrict__ alpha, const double* __restrict__ X,
                                 double* __restrict__ Y) {
  const long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (t >= static_cast<long long>(n) * nrhs) return;
  Y[t] = alpha[t / n] * X[t];
}

namespace {
inline unsigned grid_for(long long work, int threads) {
  long long g = (work + threads - 1) / threads;
  return static_cast<unsigned>(g < 1 ? 1 : g);
}
}  // namespace

int solve_block_rows() { return kRB; }
int solve_rhs_chunk() { return kRhsChunk; }
int solve_tiny_rows() { return kTinyRows; }
int solve_ancestor_chunks(int m, int np) { return ancestor_chunks(m, np); }

cudaError_t solve_max_resident(int device, int* fwd_ctas, int* bwd_ctas) {
  int sms = 0, a = 0, b = 0;
  cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(forward_pipelined_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(kSolveSmem));
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(backward_pipelined_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(kSolveSmem));
  if (e != cudaSuccess) return e;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, forward_pipelined_kernel, kST, kSolveSmem);
  if (e != cudaSuccess) return e;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, backward_pipelined_kernel, kST, kSolveSmem);
  if (e != cudaSuccess) return e;
  *fwd_ctas = a * sms;
  *bwd_ctas = b * sms;
  return cudaSuccess;
}

cudaError_t launch_forward_pipelined(const FrontDesc* fronts, const ChildLink* links, const FrontState* st,
                                     const SolvePlan& p, int task0, int ntasks, int nchunks, int grid, int epoch,
                                     int* err, unsigned long long wait_ns, int nrhs, int c0, const double* Bp, int n,
                                     cudaStream_t stream) {
  if (ntasks <= 0) return cudaSuccess;
  void* args[] = {(void*)&fronts, (void*)&links, (void*)&st, (void*)&p, (void*)&task0, (void*)&ntasks, (void*)&nchunks,
                  (void*)&epoch, (void*)&err, (void*)&wait_ns, (void*)&nrhs, (void*)&c0, (void*)&Bp, (void*)&n};
  return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(forward_pipelined_kernel), dim3(grid), dim3(kST),
                                     args, kSolveSmem, stream);
}

cudaError_t launch_backward_pipelined(const FrontDesc* fronts, const FrontState* st, const SolvePlan& p, int task0,
                                      int ntasks, int nchunks, int grid, int epoch, int* err,
                                      unsigned long long wait_ns, int nrhs, int c0, double* X, int n,
                                      cudaStream_t stream) {
  if (ntasks <= 0) return cudaSuccess;
  void* args[] = {(void*)&fronts, (void*)&st, (void*)&p, (void*)&task0, (void*)&ntasks, (void*)&nchunks, (void*)&epoch,
                  (void*)&err, (void*)&wait_ns, (void*)&nrhs, (void*)&c0, (void*)&X, (void*)&n};
  return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(backward_pipelined_kernel), dim3(grid), dim3(kST),
                                     args, kSolveSmem, stream);
}

__global__ void validate_solve_kernel(const FrontDesc* __restrict__ fronts, const FrontState* __restrict__ st,
                                      SolvePlan pl, int nfwd, int nbwd, CheckWord* chk) {
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  const auto tiny_ok = [&](int4 tk, int t) {
    if (!check(tiny_task_ok(tk.x, tk.z, pl.ntiny), chk, kChkSolveTask, t)) return;
    for (int k = 0; k < tk.z; ++k) {
      const int s = pl.tiny[tk.x + k];
      if (check(in_range(s, 0, pl.nfronts), chk, kChkSolveTask, t)) check(fronts[s].m <= kTinyRows, chk, kChkSolveTask, t);
    }
  };
  for (int s = t0; s < pl.nfronts; s += step) {
    check(in_range(pl.bwd_wait[s], -1, pl.nfronts) && pl.fwd_need[s] >= 0 && pl.bwd_need[s] >= 0 &&
              in_range(fronts[s].parent, -1, pl.nfronts) && pl.flag_base[s] >= 0 &&
              (fronts[s].m + kRB - 1) / kRB <= pl.nflags - pl.flag_base[s],
          chk, kChkSolveTable, s);
  }
  for (int t = t0; t < nfwd; t += step) {
    const int4 tk = pl.fwd_tasks[t];
    if (tk.y == -2)
      tiny_ok(tk, t);
    else if (check(in_range(tk.x, 0, pl.nfronts), chk, kChkSolveTask, t))
      check(block_task_ok(tk.y, fronts[tk.x].m, kRB, pl.flag_base[tk.x], pl.nflags), chk, kChkSolveTask, t);
  }
  for (int t = t0; t < nbwd; t += step) {
    const int4 tk = pl.bwd_tasks[t];
    if (tk.y == -2)
      tiny_ok(tk, t);
    else if (check(in_range(tk.x, 0, pl.nfronts), chk, kChkSolveTask, t) && tk.y != -1)
      check(block_task_ok(tk.y, st[tk.x].npiv, kRB, pl.flag_base[tk.x], pl.nflags) &&
                part_task_ok(tk.z, tk.w >> 20, tk.w & ((1 << 20) - 1), pl.nslots),
            chk, kChkSolveTask, t);
  }
}

void launch_validate_solve(const FrontDesc* fronts, const FrontState* st, const SolvePlan& p, int nfwd, int nbwd,
                           CheckWord* chk, cudaStream_t stream) {
  const int work = std::max({p.nfronts, nfwd, nbwd});
  if (work <= 0) return;
  validate_solve_kernel<<<std::min((work + 255) / 256, 1184), 256, 0, stream>>>(fronts, st, p, nfwd, nbwd, chk);
}

void launch_permute_in(int n, int nrhs, const int* perm, const double* B, int ldb, double* Bp, cudaStream_t stream,
                       CheckWord* chk) {
  permute_in_kernel<<<grid_for(static_cast<long long>(n) * nrhs, 256), 256, 0, stream>>>(n, nrhs, perm, B, ldb, Bp,
                                                                                         chk);
}
void launch_permute_out(int n, int nrhs, const int* perm, const double* X, double* Xout, int ldx, cudaStream_t stream,
                        CheckWord* chk) {
  permute_out_kernel<<<grid_for(static_cast<long long>(n) * nrhs, 256), 256, 0, stream>>>(n, nrhs, perm, X, Xout, ldx,
                                                                                          chk);
}
void launch_residual(int n, int nrhs, const int* rowptr, const int* colind, const int* vidx, const double* vals,
                     const double* X, int ldx, const double* B, int ldb, double* R, cudaStream_t stream) {
  residual_kernel<<<grid_for(static_cast<long long>(n) * nrhs, 256), 256, 0, stream>>>(n, nrhs, rowptr, colind, vidx,
                                                                                       vals, X, ldx, B, ldb, R);
}
void launch_absmax(const double* v, long long len, double* out, cudaStream_t stream) {
  if (len <= 0) return;
  long long g = (len + 255) / 256;
  if (g > 1184) g = 1184;
  absmax_kernel<<<static_cast<unsigned>(g), 256, 0, stream>>>(v, len, out);
}
void launch_rowsum_max(int n, const int* srowptr, const int* svidx, const double* vals, double* out,
                       cudaStream_t stream) {
  if (n <= 0) return;
  rowsum_max_kernel<<<grid_for(n, 256), 256, 0, stream>>>(n, srowptr, svidx, vals, out);
}
void launch_axpy(long long len, const double* dx, double* x, cudaStream_t stream) {
  if (len <= 0) return;
  axpy_kernel<<<grid_for(len, 256), 256, 0, stream>>>(len, dx, x);
}
int multi_dot_blocks(int n) { return static_cast<int>(std::min<long long>((n + 255) / 256, 296)); }
void launch_multi_dot(int n, int nrhs, int nvec, const double* V, long long vs, const double* W, double* partial,
                      cudaStream_t stream) {
  if (n <= 0 || nrhs <= 0 || nvec <= 0) return;
  multi_dot_kernel<<<dim3(multi_dot_blocks(n), nrhs, nvec), 256, 0, stream>>>(n, nrhs, V, vs, W, partial);
}
void launch_multi_axpy(int n, int nrhs, int nvec, const double* V, long long vs, const double* coef, double* W,
                       cudaStream_t stream) {
  if (n <= 0 || nrhs <= 0 || nvec <= 0) return;
  multi_axpy_kernel<<<grid_for(static_cast<long long>(n) * nrhs, 256), 256, 0, stream>>>(n, nrhs, nvec, V, vs, coef,
                                                                                        W);
}
void launch_col_scale(int n, int nrhs, const double* alpha, const double* X, double* Y, cudaStream_t stream) {
  if (n <= 0 || nrhs <= 0) return;
  col_scale_kernel<<<grid_for(static_cast<long long>(n) * nrhs, 256), 256, 0, stream>>>(n, nrhs, alpha, X, Y);
}

void launch_copy2d(int rows, int cols, const double* src, int lds, double* dst, int ldd, cudaStream_t stream) {
  if (rows <= 0 || cols <= 0) return;
  copy2d_kernel<<<grid_for(static_cast<long long>(rows) * cols, 256), 256, 0, stream>>>(rows, cols, src, lds, dst, ldd);
}

}  // namespace symla_gpu
