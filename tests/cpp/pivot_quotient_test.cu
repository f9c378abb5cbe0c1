// pivot_reciprocal, pivot_extreme and pivot_quotient (panel_block.cuh) against the division:
// over all exponents, and the edges of the ranges where the reciprocal is
// no longer good. Prints the largest errors; exits non-zero when one
// is above its bound.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <limits>
#include <vector>

#include "panel_block.cuh"

__global__ void quotients(int n, const double* a, const double* d, double* q, double* inv) {
  for (int i = 0; i < n; ++i) {  // one thread: the branches on d are meant to be uniform
    inv[i] = symla_gpu::pivot_reciprocal(d[i]);
    q[i] = symla_gpu::pivot_quotient(a[i], d[i], inv[i], symla_gpu::pivot_extreme(d[i]));
  }
}

static uint64_t state = 88172645463325252ull;
static uint64_t rnd() {
  state ^= state << 13;
  state ^= state >> 7;
  return state ^= state << 17;
}
static double random_double(int e0, int e1) {
  const double m = 1.0 + static_cast<double>(rnd() >> 12) * 0x1p-52;
  return std::ldexp((rnd() & 1) ? m : -m, e0 + static_cast<int>(rnd() % static_cast<uint64_t>(e1 - e0 + 1)));
}
static double ulp(double x) {
  const double m = std::fabs(x);
  return m < 0x1p-1022 ? 0x1p-1074 : std::ldexp(1.0, std::ilogb(m) - 52);
}

int main() {
  const double inf = std::numeric_limits<double>::infinity(), nan = std::numeric_limits<double>::quiet_NaN();
  std::vector<double> a, d;
  for (int i = 0; i < 40000; ++i) {  // ordinary pivots
    a.push_back(random_double(-40, 40));
    d.push_back(random_double(-40, 40));
  }
  const size_t ordinary = a.size();
  for (int i = 0; i < 40000; ++i) {  // every exponent, subnormals among them
    a.push_back(random_double(-1074, 1023));
    d.push_back(random_double(-1074, 1023));
  }
  std::vector<double> edge = {0.0, 0x1p-1074, 0x1.8p-1074, 0x1p-1026, 0x1p-1024, 0x1.8p-1024, 0x1p-1022, 5.6e-309,
                              0x1p-961, 0x1.fffffffffffffp-961, 0x1p-960, 0x1p-959, 1e-300, 1e-20, 1.0,
                              0x1.fffffffffffffp0, 3.0, 1e20, 0x1.fffffffffffffp960, 0x1p961, 1e300, 0x1p1022,
                              std::numeric_limits<double>::max(), inf, nan};
  const size_t k = edge.size();
  for (size_t i = 0; i < k; ++i) edge.push_back(-edge[i]);
  for (double x : edge)
    for (double y : edge) {
      a.push_back(x);
      d.push_back(y);
    }
  const int n = static_cast<int>(a.size());
  double* p[4];
  for (auto& x : p)
    if (cudaMalloc(&x, n * sizeof(double)) != cudaSuccess) return 2;
  cudaMemcpy(p[0], a.data(), n * sizeof(double), cudaMemcpyHostToDevice);
  cudaMemcpy(p[1], d.data(), n * sizeof(double), cudaMemcpyHostToDevice);
  quotients<<<1, 1>>>(n, p[0], p[1], p[2], p[3]);
  std::vector<double> q(n), inv(n);
  cudaMemcpy(q.data(), p[2], n * sizeof(double), cudaMemcpyDeviceToHost);
  if (cudaMemcpy(inv.data(), p[3], n * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  int bad = 0;
  size_t same = 0;
  double worst = 0.0, worst_inv = 0.0;
  for (int i = 0; i < n; ++i) {
    const double want = a[i] / d[i];
    bool ok;
    if (std::isnan(want)) {
      ok = std::isnan(q[i]);
    } else if (std::isinf(want) || std::fabs(want) >= 0x1.ffffffffffffep1023) {
      // (the residual of an infinite product is a NaN; the largest finite
      // numbers may round over)
      ok = !std::isfinite(q[i]) || std::fabs(q[i]) >= 0x1.ffffffffffffep1023;
    } else {
      // the product's two roundings, where the residual of a numerator near
      // the smallest numbers is lost; half an ulp and a little otherwise
      const double err = std::fabs(q[i] - want) / ulp(want), bound = std::fabs(a[i]) < 0x1p-900 ? 2.0 : 1.0;
      ok = err <= bound;
      worst = std::fmax(worst, err);
      if (static_cast<size_t>(i) < ordinary) {
        same += q[i] == want;
        worst_inv = std::fmax(worst_inv, std::fabs(inv[i] - 1.0 / d[i]) / ulp(1.0 / d[i]));
      }
    }
    if (!ok && ++bad <= 10) std::printf("a %a d %a: %a, division %a\n", a[i], d[i], q[i], want);
  }
  const double share = static_cast<double>(same) / static_cast<double>(ordinary);
  std::printf("worst quotient %.2f ulp, reciprocal %.2f ulp, same as the division %.6f, bad %d\n", worst, worst_inv, share, bad);
  return bad || worst_inv > 1.0 || share < 0.999 ? 1 : 0;
}
