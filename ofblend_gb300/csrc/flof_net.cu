// flof_net.cu -- kernels of the learned warm start: a small 4D convolutional
// encoder-decoder that predicts the coarsest-level deformation of the
// multiscale solve from the two coarse inputs.  It has no counterpart in
// the reference; the plain solve stays the drop-in and judges its output.
//
// Tensors are channels-last: element (v, c) of a tensor with C channels over
// a cubic 4D grid of extent R sits at v * C + c, v = x + R(y + R(z + R t)).
// The 3^4 convolutions are in flof_conv_tc.cu; here are the 1^4 output layer
// with its loss, the upsampling concatenation, the optimiser and the network
// input.  The weights are the BF16-rounded copy of the FP32 master weights
// (stored as floats); products are accumulated in FP32 with fused
// multiply-adds.  The layers are a chain of short launches: every kernel
// starts under programmatic stream serialisation.
#include <cuda_bf16.h>
#include <float.h>

#include <algorithm>

#include "flof_kernels.h"

namespace flof {

namespace {

constexpr int HI = NET_HEAD_IN, HO = NET_HEAD_OUT;
constexpr int HN = HI * HO + HO;  // parameters of the output layer
constexpr int HT = 256;           // threads of its kernels

// out[v] = W^T in[v] + b, products added in channel order
__device__ __forceinline__ float4 head_value(const float (&a)[HI], const float4 *w) {
  float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int c = 0; c < HI; ++c) {
    o.x = __fmaf_rn(a[c], w[c].x, o.x);
    o.y = __fmaf_rn(a[c], w[c].y, o.y);
    o.z = __fmaf_rn(a[c], w[c].z, o.z);
    o.w = __fmaf_rn(a[c], w[c].w, o.w);
  }
  return make_float4(o.x + w[HI].x, o.y + w[HI].y, o.z + w[HI].z, o.w + w[HI].w);
}
__device__ __forceinline__ void head_row(const float *__restrict__ in, uint32_t v,
                                         float (&a)[HI]) {
#pragma unroll
  for (int c = 0; c < HI / 4; ++c) {
    const float4 q = __ldg(reinterpret_cast<const float4 *>(in) + (size_t)v * (HI / 4) + c);
    a[4 * c] = q.x, a[4 * c + 1] = q.y, a[4 * c + 2] = q.z, a[4 * c + 3] = q.w;
  }
}
// the HI weight rows and the bias, to shared memory
__device__ __forceinline__ void head_weights(const float *__restrict__ wb, float4 *w) {
  if (threadIdx.x < HN) reinterpret_cast<float *>(w)[threadIdx.x] = __ldg(wb + threadIdx.x);
  __syncthreads();
}

__global__ void __launch_bounds__(HT)
k_head_fwd(const float *__restrict__ in, const float *__restrict__ wb, float *__restrict__ out,
           uint32_t V) {
  __shared__ float4 w[HI + 1];
  pdl_wait();
  pdl_launch_dependents();
  head_weights(wb, w);
  for (uint32_t v = blockIdx.x * HT + threadIdx.x; v < V; v += gridDim.x * HT) {
    float a[HI];
    head_row(in, v, a);
    reinterpret_cast<float4 *>(out)[v] = head_value(a, w);
  }
}

// One pass over the output layer: its value, e = value - target, the squared
// error, the gradient 2 e / n of the input behind its ReLU, and the weight
// and bias gradients.  Each thread accumulates its voxels' HN products; a
// warp adds them by the butterfly with offsets 16, 8, 4, 2, 1, in which each
// exchange also halves the number of sums a lane holds (62 exchanges instead
// of five for each of 64 sums, the same additions).  Bound by latency at 16^4
// (one voxel per thread, then the sums): 9.8 us; as separate passes (forward
// product, error, weight gradient, input gradient, mask) 40 us of kernels and
// five launches more.
__global__ void __launch_bounds__(HT, 2)
k_head_grad(const float *__restrict__ in, const float *__restrict__ wb,
            const float *__restrict__ target, float *__restrict__ din,
            double *__restrict__ part, uint32_t V, float inv) {
  __shared__ float red[HT / 32][HN];
  __shared__ double shd[HT / 32];
  __shared__ float4 w[HI + 1];
  pdl_wait();
  pdl_launch_dependents();
  head_weights(wb, w);
  float acc[HI * HO], bsum[HO] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int j = 0; j < HI * HO; ++j) acc[j] = 0.f;
  double loss = 0.0;
  for (uint32_t v = blockIdx.x * HT + threadIdx.x; v < V; v += gridDim.x * HT) {
    float a[HI];
    head_row(in, v, a);
    const float4 t = __ldg(reinterpret_cast<const float4 *>(target) + v);
    const float4 o = head_value(a, w);
    const float e[HO] = {o.x - t.x, o.y - t.y, o.z - t.z, o.w - t.w};
    float d[HO];
#pragma unroll
    for (int c = 0; c < HO; ++c) {
      loss += (double)e[c] * e[c];
      d[c] = e[c] * inv;
      bsum[c] += d[c];
    }
#pragma unroll
    for (int q = 0; q < HI / 4; ++q) {
      float g[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int ci = 4 * q + k;
        float x = __fmaf_rn(d[0], w[ci].x, 0.f);
        x = __fmaf_rn(d[1], w[ci].y, x);
        x = __fmaf_rn(d[2], w[ci].z, x);
        x = __fmaf_rn(d[3], w[ci].w, x);
        g[k] = a[ci] > 0.f ? x : 0.f;
#pragma unroll
        for (int co = 0; co < HO; ++co) acc[ci * HO + co] = acc[ci * HO + co] + a[ci] * d[co];
      }
      reinterpret_cast<float4 *>(din)[(size_t)v * (HI / 4) + q] =
          make_float4(g[0], g[1], g[2], g[3]);
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // after the exchange at offset o a lane holds the sums whose index bits
  // from the top agree with its lane bits 4, 3, ... : sum j ends in the lane
  // with lane bits (j >> 5, ..., j >> 1)
#pragma unroll
  for (int o = 16, n = HI * HO / 2; o > 0; o >>= 1, n >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int j = 0; j < n; ++j) {
      const float keep = up ? acc[j + n] : acc[j];
      const float give = up ? acc[j] : acc[j + n];
      acc[j] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  static_assert(HI * HO == 64, "two sums are left per lane");
  red[warp][2 * lane] = acc[0];
  red[warp][2 * lane + 1] = acc[1];
#pragma unroll
  for (int c = 0; c < HO; ++c) {
    float x = bsum[c];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane == 0) red[warp][HI * HO + c] = x;
  }
  loss = block_sum<HT>(loss, shd);  // synchronises the block
  if (threadIdx.x == 0) part[blockIdx.x] = loss;
  float *pf = reinterpret_cast<float *>(part + gridDim.x);
  for (int j = threadIdx.x; j < HN; j += HT) {
    float x = 0.f;
    for (int q = 0; q < HT / 32; ++q) x += red[q][j];
    pf[(size_t)blockIdx.x * HN + j] = x;
  }
}

// The blocks' partials: one warp per entry (the last warp: the loss), lane l
// adds blocks l, l + 32, ... in order, then a fixed butterfly
__global__ void k_head_sums(const double *__restrict__ part, int nblocks,
                            float *__restrict__ grad, double *__restrict__ loss, double n,
                            int acc) {
  pdl_wait();
  pdl_launch_dependents();
  const int j = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (j > HN) return;
  if (j == HN) {
    double s = 0.0;
    for (int b = lane; b < nblocks; b += 32) s += part[b];
    s = warp_sum(s);
    if (lane == 0) *loss = acc ? *loss + s / n : s / n;
    return;
  }
  const float *pf = reinterpret_cast<const float *>(part + nblocks);
  float x = 0.f;
  for (int b = lane; b < nblocks; b += 32) x += pf[(size_t)b * HN + j];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  if (lane == 0) grad[j] = acc ? grad[j] + x : x;
}

// out[v][0:c1] = lo[parent(v)][.], out[v][c1:c1+c2] = skip[v][.]; one thread
// per four channels.  Bound by its writes; with a 64-bit division per element
// it took 21 us for 48 channels at 16^4, now 7.8.
__global__ void __launch_bounds__(256)
k_upcat(const float4 *__restrict__ lo, const float4 *__restrict__ skip, float4 *__restrict__ out,
        uint32_t n, FastDiv fc, FastDiv fr, uint32_t c1, uint32_t c2) {
  pdl_wait();
  pdl_launch_dependents();
  const uint32_t R = fr.d, Rl = R / 2;
  for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    const uint32_t v = fc.div(e), c = e - v * fc.d;
    if (c < c1) {
      const uint32_t q1 = fr.div(v), q2 = fr.div(q1), t = fr.div(q2);
      const uint32_t x = v - q1 * R, y = q1 - q2 * R, z = q2 - t * R;
      const uint32_t p = x / 2 + Rl * (y / 2 + Rl * (z / 2 + Rl * (t / 2)));
      out[e] = __ldg(lo + (size_t)p * c1 + c);
    } else {
      out[e] = __ldg(skip + (size_t)v * c2 + (c - c1));
    }
  }
}

// dlo[p][c] = sum over p's 16 children in order, zero where lo is not
// positive (its ReLU); one thread per four channels, its 16 loads in flight
__global__ void __launch_bounds__(256)
k_upcat_bwd(const float4 *__restrict__ dout, const float4 *__restrict__ lo,
            float4 *__restrict__ dlo, uint32_t n, FastDiv fc1, FastDiv frl, uint32_t C) {
  pdl_wait();
  pdl_launch_dependents();
  const uint32_t Rl = frl.d, R = 2 * Rl;
  for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    const uint32_t p = fc1.div(e), c = e - p * fc1.d;
    const uint32_t q1 = frl.div(p), q2 = frl.div(q1), t = frl.div(q2);
    const uint32_t x = p - q1 * Rl, y = q1 - q2 * Rl, z = q2 - t * Rl;
    const float4 *src = dout + (size_t)(2 * x + R * (2 * y + R * (2 * z + R * 2 * t))) * C + c;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const uint32_t off = (q & 1) + R * (((q >> 1) & 1) + R * (((q >> 2) & 1) + R * (q >> 3)));
      const float4 d = __ldg(src + (size_t)off * C);
      s.x += d.x, s.y += d.y, s.z += d.z, s.w += d.w;
    }
    const float4 y4 = __ldg(lo + e);
    dlo[e] = make_float4(y4.x > 0.f ? s.x : 0.f, y4.y > 0.f ? s.y : 0.f, y4.z > 0.f ? s.z : 0.f,
                         y4.w > 0.f ? s.w : 0.f);
  }
}

// Adam on FP32 master weights, then the BF16-rounded working copy
__global__ void k_adam(float *__restrict__ w, float *__restrict__ wq, const float *__restrict__ gsum,
                       float *__restrict__ m, float *__restrict__ v, long long n, float lr,
                       float b1, float b2, float eps, float c1, float c2, float gscale) {
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
       q += (long long)gridDim.x * blockDim.x) {
    const float gr = gsum[q] * gscale;
    const float mm = b1 * m[q] + (1.f - b1) * gr;
    const float vv = b2 * v[q] + (1.f - b2) * gr * gr;
    m[q] = mm;
    v[q] = vv;
    const float upd = (mm / c1) / (sqrtf(vv / c2) + eps);
    const float nw = w[q] - lr * upd;
    w[q] = nw;
    wq[q] = __bfloat162float(__float2bfloat16_rn(nw));
  }
}

__global__ void k_round_bf16(const float *__restrict__ w, float *__restrict__ wq, long long n) {
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
       q += (long long)gridDim.x * blockDim.x)
    wq[q] = __bfloat162float(__float2bfloat16_rn(w[q]));
}

// Network input from the coarse level: channels (i0, i1) scaled by `scale`
__global__ void k_net_input(const float *__restrict__ i0, const float *__restrict__ i1,
                            float *__restrict__ x, long long V, float scale) {
  pdl_wait();
  pdl_launch_dependents();
  for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < V;
       v += (long long)gridDim.x * blockDim.x) {
    x[2 * v] = __ldg(i0 + v) * scale;
    x[2 * v + 1] = __ldg(i1 + v) * scale;
  }
}

}  // namespace

// ---- launchers --------------------------------------------------------------

static unsigned head_blocks(long long V) {
  return (unsigned)std::max(1LL, std::min((V + HT - 1) / HT, 2LL * sm_count()));
}

void net_head_fwd(const float *in, const float *wb, float *out, long long V, cudaStream_t s) {
  launch_pdl(k_head_fwd, (unsigned)grid_for(V, HT), HT, s, in, wb, out, (uint32_t)V);
}
size_t net_head_work(long long V) { return (size_t)head_blocks(V) * (1 + (HN + 1) / 2); }
void net_head_grad(const float *in, const float *wb, const float *target, float *din, float *grad,
                   double *loss, double *part, long long V, int acc, cudaStream_t s) {
  const unsigned nb = head_blocks(V);
  const double n = (double)V * HO;
  launch_pdl(k_head_grad, nb, HT, s, in, wb, target, din, part, (uint32_t)V, (float)(2.0 / n));
  launch_pdl(k_head_sums, (unsigned)(HN + 1 + 3) / 4, 128, s, (const double *)part, (int)nb, grad,
             loss, n, acc);
}

void net_upcat(const float *lo, const float *skip, float *out, int R, int c1, int c2,
               cudaStream_t s) {
  const uint32_t n = (uint32_t)((long long)R * R * R * R * (c1 + c2) / 4);
  launch_pdl(k_upcat, (unsigned)grid_for(n, 256), 256, s, (const float4 *)lo,
             (const float4 *)skip, (float4 *)out, n, FastDiv((c1 + c2) / 4), FastDiv(R),
             (uint32_t)c1 / 4, (uint32_t)c2 / 4);
}
void net_upcat_bwd(const float *dout, const float *lo, float *dlo, int R, int c1, int c2,
                   cudaStream_t s) {
  const long long rl = R / 2;
  const uint32_t n = (uint32_t)(rl * rl * rl * rl * c1 / 4);
  launch_pdl(k_upcat_bwd, (unsigned)grid_for(n, 256), 256, s, (const float4 *)dout,
             (const float4 *)lo, (float4 *)dlo, n, FastDiv(c1 / 4), FastDiv((uint32_t)rl),
             (uint32_t)(c1 + c2) / 4);
}
void net_adam(float *w, float *wq, const float *g, float *m, float *v, long long n, float lr,
              int step, float gscale, cudaStream_t s) {
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
  k_adam<<<grid_for(n, 256), 256, 0, s>>>(w, wq, g, m, v, n, lr, b1, b2, eps, c1, c2, gscale);
}
void net_round_bf16(const float *w, float *wq, long long n, cudaStream_t s) {
  k_round_bf16<<<grid_for(n, 256), 256, 0, s>>>(w, wq, n);
}
void net_input(const float *i0, const float *i1, float *x, long long V, float scale,
               cudaStream_t s) {
  launch_pdl(k_net_input, (unsigned)grid_for(V, 256), 256, s, i0, i1, x, V, scale);
}

}  // namespace flof
