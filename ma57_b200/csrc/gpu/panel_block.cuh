// The two halves of an unpivoted panel of at most 32 pivots, shared by the
// static and the speculative panel kernels: the diagonal block's LDL^T by one
// warp, and the rows below it.
#pragma once

#include "common.cuh"

namespace symla_gpu {

constexpr int kPanelMax = 32;    // pivots per panel
constexpr int kBlkStride = 34;   // even: pairs of a row are one 16-byte load

// The diagonal block in shared memory. In: db's lower triangle, the block's
// current values. Out: L below the diagonal of db (d on it); wv[i][c] = the
// current value of row i in column c before scaling, d_c L(i, c); d, 1 / d
// and the applied perturbation; extreme: some d is (pivot_extreme).
struct alignas(16) DiagBlock {
  double db[kPanelMax][kBlkStride];
  double wv[kPanelMax][kBlkStride];
  double dv[kPanelMax], iv[kPanelMax], pv[kPanelMax];
  int extreme;
};

// Static pivoting (dense_kernel.hpp:982-1034): the pivot that replaces akk,
// without a branch, and what that adds to it. Only a pivot that fails the floor
// test is replaced; a NaN, or an infinite one of the right sign, is left alone
// and has nothing added (the difference of the two would be a NaN).
__device__ __forceinline__ double static_pivot(double akk, int sign, double floorv, double delta, double& applied) {
  const double t = sign == 0 ? fabs(akk) : (sign > 0 ? akk : -akk);
  const bool up = sign > 0 || (sign == 0 && akk >= 0.0);
  const bool need = t < floorv;
  const double d = need ? akk + (up ? delta : -delta) : akk;
  applied = need ? d - akk : 0.0;
  return d;
}

// A pivot outside [2^-960, 2^960): there 1 / d, or a step towards it, would
// overflow or lose bits to underflow (1 / d is infinite below 2^-1024), and what
// follows takes the division instead. Uniform: every lane has the same pivot.
__device__ __forceinline__ bool pivot_extreme(double d) {
  const unsigned e = (static_cast<unsigned>(__double2hiint(d)) >> 20) & 0x7ff;
  return e - (1023 - 960) >= 2 * 960;
}

// 1 / d by Newton's iteration, r <- r + r (1 - d r), two steps from the
// hardware's approximation: under one ulp off. Not for an extreme d.
__device__ __forceinline__ double pivot_reciprocal(double d) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
  r = fma(r, fma(-d, r, 1.0), r);
  return fma(r, fma(-d, r, 1.0), r);
}

// a / d from inv = 1 / d: the product, corrected by one residual (Markstein's
// quotient, IBM J. Res. Dev. 34(1), 1990). The product alone would be off by the
// reciprocal's relative error in the whole column, and the updates (which take
// L D as the values before the division) would carry it into the whole Schur
// complement. Not for an extreme d. (An infinite quotient comes out as a NaN.)
__device__ __forceinline__ double pivot_quotient(double a, double d, double inv) {
  const double q = a * inv;
  return fma(fma(-q, d, a), inv, q);
}

// a / d for any d, extreme = pivot_extreme(d) (a call, so that the division
// stays out of the loops over pivots).
static __device__ __noinline__ double pivot_divide(double a, double d) { return a / d; }
__device__ __forceinline__ double pivot_quotient(double a, double d, double inv, bool extreme) {
  return extreme ? pivot_divide(a, d) : pivot_quotient(a, d, inv);
}

// LDL^T of the np x np block by one warp, lane = row, in steps of eight
// columns: the step's columns of the lane's row are brought up to date from
// the earlier steps (left-looking, the row's values in registers, eight
// independent sums), then every lane factors the 8 x 8 diagonal block
// redundantly in registers while it eliminates its own row. No shuffle, and
// one warp barrier per column instead of two. Products are summed
// apart and subtracted from an entry once per step: subtracting them one by
// one would round each time at the size of the entry, which on a diagonally
// heavy matrix is far above that of the sum. Entries past np are garbage of
// which no row or column below np depends.
//
// What bounds it is the chain of 32 reciprocals, each followed by the update of the
// next pivot (one warp, 255 registers allowed). Column by column, with the
// row in shared memory, a column took 890 cycles (14 us per block); now it
// takes about 260 (keeping the sums apart costs the 64^3 stencil's panels 0.4
// of 31 ms, the quotients' residual step 0.9).
//
// Returns (in every lane) whether a pivot was extreme: the block is then to be
// staged anew and given to factor_diag_block_divide.
template <bool Static>
__device__ __forceinline__ bool factor_diag_block(DiagBlock& B, int np, int lane, int lane_sign, double floorv,
                                                  double delta) {
  double a[kPanelMax];  // the lane's row: values before scaling, by column
#pragma unroll
  for (int j0 = 0; j0 < kPanelMax; j0 += 8) {
    if (j0 >= np) break;
    double x[8], xs[8];  // the lane's row: values at the step's start, the step's sums
#pragma unroll
    for (int c = 0; c < 8; ++c) xs[c] = 0.0;
#pragma unroll
    for (int t = 0; t < j0; t += 2)
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const double2 l = *reinterpret_cast<const double2*>(&B.db[j0 + c][t]);
        xs[c] = fma(a[t], l.x, xs[c]);
        xs[c] = fma(a[t + 1], l.y, xs[c]);
      }
#pragma unroll
    for (int c = 0; c < 8; c += 2) {
      const double2 v = *reinterpret_cast<const double2*>(&B.db[lane][j0 + c]);
      x[c] = v.x - xs[c];
      x[c + 1] = v.y - xs[c + 1];
      xs[c] = xs[c + 1] = 0.0;
    }
    if (lane >= j0 && lane < j0 + 8)
#pragma unroll
      for (int c = 0; c < 8; ++c) B.db[lane][j0 + c] = x[c];
    __syncwarp();
    double U[8][8];  // sums of the 8 x 8 block's entries
    double T[8];     // the pivot column's values
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      T[r] = B.db[j0 + r][j0];
#pragma unroll
      for (int c = 0; c <= r; ++c) U[r][c] = 0.0;
    }
    int sign[8];
    if (Static)
#pragma unroll
      for (int c = 0; c < 8; ++c) sign[c] = __shfl_sync(0xffffffffu, lane_sign, j0 + c);
    __syncwarp();
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int col = j0 + c;
      double next[8];  // the next column's values at the step's start
#pragma unroll
      for (int r = c + 1; r < 8; ++r) next[r] = B.db[j0 + r][col + 1];
      if (c < 7) __syncwarp();  // every lane has read column col + 1 before any stores its L there
      const double akk = T[c];
      double d = akk, applied = 0.0;
      if (Static) d = static_pivot(akk, sign[c], floorv, delta, applied);
      const double inv = pivot_reciprocal(d);
      double l[8];
#pragma unroll
      for (int r = c + 1; r < 8; ++r) l[r] = pivot_quotient(T[r], d, inv);
#pragma unroll
      for (int r2 = c + 1; r2 < 8; ++r2)
#pragma unroll
        for (int r = r2; r < 8; ++r) U[r][r2] = fma(T[r], l[r2], U[r][r2]);
      const double v = x[c] - xs[c];
      a[col] = v;
#pragma unroll
      for (int c2 = c + 1; c2 < 8; ++c2) xs[c2] = fma(v, l[c2], xs[c2]);
#pragma unroll
      for (int r = c + 1; r < 8; ++r) T[r] = next[r] - U[r][c + 1];
      // every lane stores: what lands above the diagonal is not read
      const double li = pivot_quotient(v, d, inv);
      B.db[lane][col] = lane == col ? d : li;
      B.wv[lane][col] = v;
      B.dv[col] = d;
      B.iv[col] = inv;
      if (Static) B.pv[col] = applied;
    }
    __syncwarp();
  }
  // (a NaN is none: what it comes from was found before it; nor, under threshold
  // pivoting, a zero, which is never accepted)
  const double own = B.dv[lane];
  const bool extreme = lane < np && pivot_extreme(own) && own == own && (Static || own != 0.0);
  const bool any = __any_sync(0xffffffffu, extreme);
  if (lane == 0) B.extreme = any;
  return any;
}

// The same with plain divisions, column by column, for a block staged anew of
// which factor_diag_block found an extreme pivot. (Rare, so small: the fast one
// is straight-line code that runs once per panel, and what is added to it is
// paid in instruction fetches. The panels of the 64^3 stencil take 40 ms with an
// extreme pivot handled where it is met, 33 with a branch per column for its
// reciprocal alone, 31 with one check at the end.)
template <bool Static>
__device__ __noinline__ void factor_diag_block_divide(DiagBlock& B, int np, int lane, int lane_sign, double floorv,
                                                      double delta) {
  __syncwarp();
#pragma unroll 1
  for (int c = 0; c < np; ++c) {
    double sum = 0.0;
#pragma unroll 1
    for (int t = 0; t < c; ++t) sum = fma(B.wv[lane][t], B.db[c][t], sum);
    const double v = B.db[lane][c] - sum;  // (lanes above the diagonal: not read)
    const double akk = __shfl_sync(0xffffffffu, v, c);
    double d = akk, applied = 0.0;
    if (Static) d = static_pivot(akk, __shfl_sync(0xffffffffu, lane_sign, c), floorv, delta, applied);
    const double l = v / d;
    __syncwarp();
    B.db[lane][c] = lane == c ? d : l;
    B.wv[lane][c] = v;
    if (lane == c) {
      B.dv[c] = d;
      if (Static) B.pv[c] = applied;
    }
    __syncwarp();
  }
}

// A row below the block: a[c] becomes the row's current value in column c,
// the raw one minus sum_t a_t L(c, t) (L = a / d), the sum formed apart in
// four parts. Columns past np are computed on garbage and not used. The loads
// of L are warp-uniform pairs. (Two rows per thread would halve them, but
// leave no registers to load ahead with: the pass then waits for every pair
// and took 10 us instead of 2.)
__device__ __forceinline__ void panel_row(const DiagBlock& B, int np, double (&a)[kPanelMax]) {
#pragma unroll
  for (int c = 1; c < kPanelMax; ++c) {
    if ((c & 7) == 0 && c >= np) break;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
#pragma unroll
    for (int t = 0; t < c; t += 2) {
      const double2 l = *reinterpret_cast<const double2*>(&B.db[c][t]);
      if (t & 2) {
        s2 = fma(a[t], l.x, s2);
        if (t + 1 < c) s3 = fma(a[t + 1], l.y, s3);
      } else {
        s0 = fma(a[t], l.x, s0);
        if (t + 1 < c) s1 = fma(a[t + 1], l.y, s1);
      }
    }
    a[c] -= (s0 + s1) + (s2 + s3);
  }
}

// Column maxima of a warp's rows: lane c returns the largest |a[c]| over the
// warp's lanes with `in` set (bit patterns of non-negative doubles order like
// the values, and a NaN wins): per column a 32-bit reduction of the high words
// and one of the low words that go with the largest.
__device__ __forceinline__ unsigned long long warp_column_max(const double (&a)[kPanelMax], bool in, int np, int lane) {
  unsigned hi = 0, lo = 0;
#pragma unroll
  for (int c = 0; c < kPanelMax; ++c) {
    if ((c & 7) == 0 && c >= np) break;
    const unsigned long long b = in ? static_cast<unsigned long long>(__double_as_longlong(fabs(a[c]))) : 0ull;
    const unsigned h = static_cast<unsigned>(b >> 32);
    const unsigned mh = __reduce_max_sync(0xffffffffu, h);
    const unsigned ml = __reduce_max_sync(0xffffffffu, h == mh ? static_cast<unsigned>(b) : 0u);
    if (lane == c) {
      hi = mh;
      lo = ml;
    }
  }
  return lane < np ? static_cast<unsigned long long>(hi) << 32 | lo : 0ull;
}

// A row's L = a / d and -(L D) = -a in the packed operands (p: pivot q0 of the
// row), and put(c, l) for every column c < np: eight columns at a time, so
// that the loads of the divisors do not wait for the stores before them.
template <class Put>
__device__ __forceinline__ void store_panel_row(const DiagBlock& B, int np, const double (&a)[kPanelMax], double* P,
                                                int64_t pw, int prt, int q0, int i, Put&& put) {
  double* p = P + packed_at(prt, q0, i);
  const int64_t next = static_cast<int64_t>(prt) * kPkTile - 16 * kPkRow;  // to the next 16-pivot chunk
#pragma unroll
  for (int c0 = 0; c0 < kPanelMax; c0 += 8) {
    if (c0 >= np) break;
    double l[8];
#pragma unroll
    for (int c = 0; c < 8; c += 2) {
      const double2 iv = *reinterpret_cast<const double2*>(&B.iv[c0 + c]);
      const double2 dv = *reinterpret_cast<const double2*>(&B.dv[c0 + c]);
      l[c] = pivot_quotient(a[c0 + c], dv.x, iv.x);
      l[c + 1] = pivot_quotient(a[c0 + c + 1], dv.y, iv.y);
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      if (c0 + c < np) {
        put(c0 + c, l[c]);
        p[0] = l[c];
        p[pw] = -a[c0 + c];
      }
      p += kPkRow;
      if (((q0 + c0 + c + 1) & 15) == 0) p += next;
    }
  }
  if (B.extreme)  // (the thread's own stores, read back)
#pragma unroll 1
    for (int c = 0; c < np; ++c) {
      double* pk = P + packed_at(prt, q0 + c, i);
      pk[0] = -pk[pw] / B.dv[c];
      put(c, pk[0]);
    }
}

}  // namespace symla_gpu
