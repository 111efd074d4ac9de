// quotient (csrc/flof_common.cuh) against the FP64 division, over the range that
// its guards admit and at their edges.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "flof_common.cuh"

__global__ void k_quotient(const double *a, const double *b, float *q, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) q[i] = flof::quotient(a[i], b[i]);
}

int main() {
  std::vector<double> a, b;
  unsigned long long s = 88172645463325252ull;
  auto rnd = [&] {  // xorshift64 (Marsaglia 2003), in [0, 1)
    s ^= s << 13;
    s ^= s >> 7;
    s ^= s << 17;
    return (double)(s >> 11) * (1.0 / 9007199254740992.0);
  };
  auto add = [&](double x, double y) {
    a.push_back(x);
    b.push_back(y);
  };
  for (int i = 0; i < 4000000; ++i) {  // every magnitude, both signs
    const double x = std::pow(10.0, 62 * rnd() - 31), y = std::pow(10.0, 62 * rnd() - 31);
    add(rnd() < 0.5 ? x : -x, rnd() < 0.5 ? y : -y);
  }
  for (int i = 0; i < 4000000; ++i) {  // like sums: ratios around one
    const double y = std::pow(10.0, 20 * rnd() - 10);
    add(y * std::pow(10.0, 4 * rnd() - 3), y);
  }
  for (int i = 0; i < 1000000; ++i) {  // quotients that are floats, or next to one
    const float q = (float)(1 + rnd()), y = (float)(1 + rnd());
    add((double)q * y * (1 + (i % 5 - 2) * 0x1p-52), y);
  }
  const double edge[] = {0.0, -0.0, 1e-30, 1e30, 1e-31, 1e31, 1e-300, 1e300, 1e-45, 3.4e38, INFINITY, -INFINITY,
                         NAN, 1.0, -3.0, 9.999999e-31, 1.0000001e-30, 9.999999e29, 1.0000001e30};
  const size_t random = a.size();
  for (double x : edge)
    for (double y : edge) add(x, y);
  const int n = (int)a.size();
  double *da, *db;
  float *dq;
  std::vector<float> q(n);
  if (cudaMalloc(&da, n * 8) || cudaMalloc(&db, n * 8) || cudaMalloc(&dq, n * 4) ||
      cudaMemcpy(da, a.data(), n * 8, cudaMemcpyHostToDevice) ||
      cudaMemcpy(db, b.data(), n * 8, cudaMemcpyHostToDevice))
    return std::printf("no device memory\n"), 1;
  k_quotient<<<(n + 255) / 256, 256>>>(da, db, dq, n);
  if (cudaMemcpy(q.data(), dq, n * 4, cudaMemcpyDeviceToHost)) return std::printf("kernel failed\n"), 1;
  int bad = 0, far = 0;
  for (int i = 0; i < n; ++i) {
    const double want = a[i] / b[i];
    const float near = (float)want;
    bool ok = std::memcmp(&q[i], &near, 4) == 0 || (std::isnan(near) && std::isnan(q[i]));
    if (!ok && std::isfinite(near) && std::fabs(want) > 1e-30) {
      // the other neighbour, where the quotient lies in the middle
      ++far;
      const double ulp = std::ldexp(1.0, std::ilogb(want) - 23);
      ok = std::fabs(q[i] - want) <= 0.5 * ulp + std::ldexp(std::fabs(want), -43);
    }
    if (!ok && bad++ < 10) std::printf("%d: %.17g / %.17g = %.9g, not %.9g\n", i, a[i], b[i], q[i], near);
  }
  std::printf("%zu random pairs, %d the other neighbour, %d wrong\n", random, far, bad);
  return bad != 0;
}
