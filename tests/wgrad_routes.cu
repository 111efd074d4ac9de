// Stride-1 weight gradients (csrc/flof_conv_tc.cu) on both sides of the rule
// that chooses between halo tiles and im2col, against FP64 on the host.
#include <cmath>
#include <cstdio>
#include <vector>

#include "flof_kernels.h"

using namespace flof;

int main() {
  struct Shape {
    int R, cin, cout;
  };
  const Shape shapes[] = {{1, 64, 64}, {2, 64, 64}, {3, 64, 64}, {4, 64, 64}, {7, 64, 64},  {9, 64, 64}, {12, 64, 64},
                          {13, 64, 64}, {2, 32, 32}, {4, 32, 32}, {10, 32, 32}, {2, 96, 32}, {5, 96, 32}, {4, 48, 16}};
  unsigned s = 7;
  auto rnd = [&] {
    s = s * 1664525u + 1013904223u;
    return (float)(s >> 8) * (2.f / 16777216.f) - 1.f;
  };
  int bad = 0;
  for (const Shape &h : shapes) {
    const int R = h.R, ci = h.cin, co = h.cout;
    const size_t V = (size_t)R * R * R * R, ng = (size_t)(81 * ci + 1) * co;
    std::vector<float> in(V * ci), dout(V * co), g(ng);
    for (float &v : in) v = rnd();
    for (float &v : dout) v = rnd();
    float *din, *ddout, *dg, *work;
    int *err;
    if (cudaMalloc(&din, in.size() * 4) || cudaMalloc(&ddout, dout.size() * 4) || cudaMalloc(&dg, ng * 4) ||
        cudaMalloc(&work, net_tc_work(R, R, ci, co, false) * 4) || cudaMalloc(&err, 4) || cudaMemset(err, 0, 4) ||
        cudaMemcpy(din, in.data(), in.size() * 4, cudaMemcpyHostToDevice) ||
        cudaMemcpy(ddout, dout.data(), dout.size() * 4, cudaMemcpyHostToDevice))
      return std::printf("no device memory\n"), 1;
    for (int acc = 0; acc < 2; ++acc) {  // written, then added to: twice the sums
      net_tc_conv_bwd_weight(din, ddout, dg, work, R, R, ci, co, 1, acc, err, 0);
      int e = 0;
      if (cudaMemcpy(g.data(), dg, ng * 4, cudaMemcpyDeviceToHost) ||
          cudaMemcpy(&e, err, 4, cudaMemcpyDeviceToHost) || e)
        return std::printf("%d^4 %d -> %d: %s, device error %d\n", R, ci, co,
                           cudaGetErrorString(cudaGetLastError()), e), 1;
      double worst = 0;
      for (int q = 0; q < 400; ++q) {
        // every tap of some channel pairs, and the bias row
        const int tap = q % 82, a = (q * 7 + q / 82) % ci, b = (q * 5 + q / 3) % co;
        const int off[4] = {tap % 3 - 1, tap / 3 % 3 - 1, tap / 9 % 3 - 1, tap / 27 - 1};
        double want = 0, size = 0;
        for (size_t v = 0; v < V; ++v) {
          int c[4] = {(int)(v % R), (int)(v / R % R), (int)(v / R / R % R), (int)(v / R / R / R)};
          double x = 1;
          if (tap < 81) {
            size_t u = 0, mul = 1;
            bool inside = true;
            for (int k = 0; k < 4; ++k) {
              const int p = c[k] + off[k];
              inside = inside && p >= 0 && p < R;
              u += p * mul;
              mul *= R;
            }
            if (!inside) continue;
            x = in[u * ci + a];
          }
          want += x * dout[v * co + b];
          size += std::fabs(x * dout[v * co + b]);
        }
        const double got = g[tap < 81 ? ((size_t)tap * ci + a) * co + b : (size_t)81 * ci * co + b];
        // operands as two BF16 parts (2^-17 each of their rounding, the product of
        // the low parts left out), sums in float
        const double tol = (1 + acc) * std::ldexp(size, -15) + 1e-12;
        worst = std::fmax(worst, std::fabs(got - (1 + acc) * want) / tol);
      }
      std::printf("%d^4 %d -> %d: %.3f of the bound\n", R, ci, co, worst);
      bad += !(worst <= 1);
    }
    cudaFree(din), cudaFree(ddout), cudaFree(dg), cudaFree(work), cudaFree(err);
  }
  std::printf(bad ? "%d outside\n" : "OK\n", bad);
  return bad != 0;
}
