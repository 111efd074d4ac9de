// Beta of the chained PCG (csrc/flof_solve.cu), which the matvec predicts from
// its sums, against the ratio of the z.r summed before and after the step that
// it belongs to.
#include <cmath>
#include <cstdio>
#include <vector>

#include "flof_kernels.h"

using namespace flof;

#define OK(x)                                                              \
  do {                                                                     \
    const cudaError_t e_ = (x);                                            \
    if (e_ != cudaSuccess) {                                               \
      std::printf("%s: %s\n", #x, cudaGetErrorString(e_));                 \
      return 1;                                                            \
    }                                                                      \
  } while (0)

int main() {
  const Dims4 d{43, 45, 41, 42};
  const size_t n = (size_t)d.cells();
  std::vector<float> h0(n), h1(n);
  unsigned s = 1;
  auto rnd = [&] {
    s = s * 1664525u + 1013904223u;
    return (float)(s >> 8) * (2.f / 16777216.f) - 1.f;
  };
  // The gradients are too small to show in g^2 + diag, which is then the same
  // number in every cell, as outside a surface's band: an error of its
  // reciprocal is common to all terms of a sum.
  for (size_t i = 0; i < n; ++i) {
    h1[i] = 1e-8f * rnd();
    h0[i] = 1e4f * rnd();
  }
  float *i0, *i1, *fpart;
  float4 *g, *r, *x, *q, *pb;
  double *dpart;
  CGState *st;
  OK(cudaMalloc(&i0, n * 4));
  OK(cudaMalloc(&i1, n * 4));
  OK(cudaMalloc(&g, n * 16));
  OK(cudaMalloc(&r, n * 16));
  OK(cudaMalloc(&x, n * 16));
  OK(cudaMalloc(&q, n * 16));
  OK(cudaMalloc(&pb, CG_RING * n * 16));
  OK(cudaMalloc(&dpart, 65536 * 8));
  OK(cudaMalloc(&fpart, 65536 * 4));
  OK(cudaMalloc(&st, sizeof(CGState)));
  OK(cudaMemset(st, 0, sizeof(CGState)));
  OK(cudaMemcpy(i0, h0.data(), n * 4, cudaMemcpyHostToDevice));
  OK(cudaMemcpy(i1, h1.data(), n * 4, cudaMemcpyHostToDevice));
  CGRing ring;
  ring.n = CG_RING;
  for (int k = 0; k < CG_RING; ++k) ring.p[k] = pb + k * n;
  const double cells = (double)(d.x - 2) * (d.y - 2) * (d.z - 2) * (d.t - 2);
  int bad = 0;
  // eight diagonals with the usual ratio of the terms, then two of a system so
  // near to its diagonal that a step leaves next to nothing of z.r
  for (int k = 0; k < 10; ++k) {
    const float smooth = k < 8 ? 0.001f * (1.f + 0.13f * k) : k == 8 ? 1e-5f : 1e-9f;
    const float energy = k < 8 ? 1e-4f : 0.01f;
    OFConsts c;
    c.mDx = 1.f / d.x;
    c.mDt = 1.f;
    c.dxf = 0.5f * d.x;
    c.wSmooth = smooth;
    c.wEnergy = energy;
    c.offd = -smooth;
    c.diag = 8.f * smooth + energy;
    OK(cudaMemset(pb, 0, CG_RING * n * 16));
    launch_of_assemble_init(i0, i1, nullptr, g, r, ring.p[0], x, d, c, 1e-20f, st, dpart, fpart, 0);
    CGState h;
    OK(cudaMemcpy(&h, st, sizeof(h), cudaMemcpyDeviceToHost));
    if (h.done != CG_RUNNING) {
      std::printf("system %d did not start (%d)\n", k, h.done);
      return 1;
    }
    for (int it = 0; it < (k < 8 ? 6 : 2); ++it) {
      const double before = h.sigma;
      launch_cg_matvec(ring.p[it % CG_RING], g, q, d, c, st, dpart, it % CG_RING, 0, CGTune());
      launch_cg_step(x, r, q, ring, it, g, i1, d, c, st, dpart, fpart, 1 << 30, 0, CGTune());
      OK(cudaMemcpy(&h, st, sizeof(h), cudaMemcpyDeviceToHost));
      const double want = h.sigma / before;
      // Four sums of 4 x cells products, together 5 (1 + beta) z.r, whose two or
      // three roundings to float are independent: the sums' error is 2^-24 over
      // the root of their number, 20 of these; then beta's rounding to float.
      const double tol = 20 * 5 * (1 + want) * std::ldexp(1.0, -24) / std::sqrt(4 * cells) +
                         std::ldexp(want, -24);
      const double err = std::fabs((double)h.betaf - want);
      std::printf("system %d step %d: beta %.6e, error %.2e of %.2e\n", k, it, want, err, tol);
      if (!(err <= tol) || h.betaf < 0.f) ++bad;
    }
  }
  std::printf(bad ? "%d outside\n" : "OK\n", bad);
  return bad != 0;
}
