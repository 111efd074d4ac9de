// flof_ops.cu -- Grid4d operations, reductions, resampling, semi-Lagrangian
// advection and the hi-res slice lookup of the FlOF path.
//
// Reference: source/grid4d.{h,cpp} (Grid4d ops, knSetBnd4d*, kn4dMax*,
// knInterpol4d), source/plugin/optflow4d.cpp (semiLagrange4d :1275,
// calcLsDiffTempl :895, knSemiLagrangeLookupSlice4d_WithVel :1648), and the
// mode-2/3 blends of scenes/flof.py (:603-610, :750-755).
#include <float.h>

#include "flof_kernels.h"

namespace flof {

// SM count of the current device, read once (thread-safe static init).
int sm_count() {
  static const int n = [] {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v > 0 ? v : 1;
  }();
  return n;
}

int current_device() {
  int dev = 0;
  cudaGetDevice(&dev);
  return dev;
}

int grid_for(long long n, int nt, int per_sm) {
  long long b = (n + nt - 1) / nt;
  long long cap = (long long)sm_count() * per_sm;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return (int)b;
}

constexpr int NT = 256;

// Blocks for a gather kernel: one trip per thread.  These kernels have 5 or 6
// resident blocks per SM, so a capped grid of 8 per SM runs as one full wave
// and a mostly empty one; with one trip per thread the SMs refill as blocks
// end.
static inline unsigned grid_all(long long n) { return (unsigned)((n + NT - 1) / NT); }

// ---------------------------------------------------------------------------
// Elementwise
// ---------------------------------------------------------------------------

// op: 0 set, 1 add, 2 mult
template <int OP>
__global__ void k_const_vec4(float4 *a, long long n, float4 v) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    float4 x = a[i];
    if (OP == 0) x = v;
    if (OP == 1) { x.x += v.x; x.y += v.y; x.z += v.z; x.w += v.w; }
    if (OP == 2) { x.x *= v.x; x.y *= v.y; x.z *= v.z; x.w *= v.w; }
    a[i] = x;
  }
}
template <int OP>
__global__ void k_const_real(float *a, long long n, float v) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    float x = a[i];
    if (OP == 0) x = v;
    if (OP == 1) x += v;
    if (OP == 2) x *= v;
    a[i] = x;
  }
}

template <int OP>
static void const_op(float *a, long long ncell, int nc, float4 v, cudaStream_t s) {
  if (ncell <= 0) return;
  if (nc == 4) {
    k_const_vec4<OP><<<grid_for(ncell, NT), NT, 0, s>>>((float4 *)a, ncell, v);
  } else if (ncell % 4 == 0 && ((uintptr_t)a & 15) == 0) {
    float4 vv = make_float4(v.x, v.x, v.x, v.x);
    k_const_vec4<OP><<<grid_for(ncell / 4, NT), NT, 0, s>>>((float4 *)a, ncell / 4, vv);
  } else {
    k_const_real<OP><<<grid_for(ncell, NT), NT, 0, s>>>(a, ncell, v.x);
  }
}
void launch_set_const(float *a, long long ncell, int nc, float4 v, cudaStream_t s) {
  const_op<0>(a, ncell, nc, v, s);
}
void launch_add_const(float *a, long long ncell, int nc, float4 v, cudaStream_t s) {
  const_op<1>(a, ncell, nc, v, s);
}
void launch_mult_const(float *a, long long ncell, int nc, float4 v, cudaStream_t s) {
  const_op<2>(a, ncell, nc, v, s);
}

// op: 0 add, 1 sub, 2 scaled add with per-component factor
template <int OP>
__global__ void k_binary_vec4(float4 *a, const float4 *__restrict__ b, long long n,
                              float4 f) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    float4 x = a[i];
    const float4 y = __ldg(b + i);
    if (OP == 0) { x.x += y.x; x.y += y.y; x.z += y.z; x.w += y.w; }
    if (OP == 1) { x.x -= y.x; x.y -= y.y; x.z -= y.z; x.w -= y.w; }
    if (OP == 2) {
      x.x += f.x * y.x; x.y += f.y * y.y; x.z += f.z * y.z; x.w += f.w * y.w;
    }
    a[i] = x;
  }
}
template <int OP>
__global__ void k_binary_real(float *a, const float *__restrict__ b, long long n,
                              float f) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    float x = a[i];
    const float y = __ldg(b + i);
    if (OP == 0) x += y;
    if (OP == 1) x -= y;
    if (OP == 2) x += f * y;
    a[i] = x;
  }
}
template <int OP>
static void binary_op(float *a, const float *b, long long nfloat, float4 f,
                      bool per_comp, cudaStream_t s) {
  if (nfloat <= 0) return;
  const bool vec = nfloat % 4 == 0 && ((uintptr_t)a & 15) == 0 && ((uintptr_t)b & 15) == 0;
  if (vec) {
    float4 ff = per_comp ? f : make_float4(f.x, f.x, f.x, f.x);
    k_binary_vec4<OP><<<grid_for(nfloat / 4, NT), NT, 0, s>>>((float4 *)a, (const float4 *)b,
                                                             nfloat / 4, ff);
  } else {
    k_binary_real<OP><<<grid_for(nfloat, NT), NT, 0, s>>>(a, b, nfloat, f.x);
  }
}
void launch_add(float *a, const float *b, long long n, cudaStream_t s) {
  binary_op<0>(a, b, n, make_float4(0, 0, 0, 0), false, s);
}
void launch_sub(float *a, const float *b, long long n, cudaStream_t s) {
  binary_op<1>(a, b, n, make_float4(0, 0, 0, 0), false, s);
}
void launch_add_scaled(float *a, const float *b, long long ncell, int nc, float4 f,
                       cudaStream_t s) {
  binary_op<2>(a, b, ncell * nc, f, nc == 4, s);
}

__global__ void __launch_bounds__(NT)
k_sub_box(float4 *__restrict__ a, const float4 *__restrict__ b, Dims4 d, BoxDecoder bx,
          uint32_t n) {
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    int i, j, k, l;
    bx.decode(q, i, j, k, l);
    const idx_t id = d.index(i, j, k, l);
    const float4 x = a[id], y = __ldg(b + id);
    a[id] = make_float4(x.x - y.x, x.y - y.y, x.z - y.z, x.w - y.w);
  }
}
void launch_sub_box(float4 *a, const float4 *b, Dims4 d, const CellBox &box, cudaStream_t s) {
  const long long n = box.cells();
  if (n == 0) return;
  const BoxDecoder bx = make_decoder(box.hi[0] - box.lo[0], box.hi[1] - box.lo[1],
                                     box.hi[2] - box.lo[2], box.lo[0], box.lo[1], box.lo[2],
                                     box.lo[3]);
  k_sub_box<<<grid_for(n, NT), NT, 0, s>>>(a, b, d, bx, (uint32_t)n);
}

// ---------------------------------------------------------------------------
// Borders (grid4d.cpp:355-407)
// ---------------------------------------------------------------------------

__global__ void k_set_bound(float *a, Dims4 d, BoxDecoder bx, int nc, float4 v,
                            int w) {
  const uint32_t n = (uint32_t)d.cells();
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < n;
       q += gridDim.x * blockDim.x) {
    int i, j, k, l;
    bx.decode(q, i, j, k, l);
    const bool b = (i <= w || i >= d.x - 1 - w || j <= w || j >= d.y - 1 - w ||
                    k <= w || k >= d.z - 1 - w || l <= w || l >= d.t - 1 - w);
    if (!b) continue;
    if (nc == 4) ((float4 *)a)[q] = v;
    else a[q] = v.x;
  }
}
void launch_set_bound(float *a, Dims4 d, int nc, float4 v, int w, cudaStream_t s) {
  BoxDecoder bx = make_decoder(d.x, d.y, d.z, 0, 0, 0, 0);
  k_set_bound<<<grid_for(d.cells(), NT), NT, 0, s>>>(a, d, bx, nc, v, w);
}

__global__ void k_set_bound_neumann(float *a, Dims4 d, BoxDecoder bx, int nc, int w) {
  const uint32_t n = (uint32_t)d.cells();
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < n;
       q += gridDim.x * blockDim.x) {
    int i, j, k, l;
    bx.decode(q, i, j, k, l);
    bool set = false;
    int si = i, sj = j, sk = k, sl = l;
    if (i <= w) { si = w + 1; set = true; }
    if (i >= d.x - 1 - w) { si = d.x - 1 - w - 1; set = true; }
    if (j <= w) { sj = w + 1; set = true; }
    if (j >= d.y - 1 - w) { sj = d.y - 1 - w - 1; set = true; }
    if (k <= w) { sk = w + 1; set = true; }
    if (k >= d.z - 1 - w) { sk = d.z - 1 - w - 1; set = true; }
    if (l <= w) { sl = w + 1; set = true; }
    if (l >= d.t - 1 - w) { sl = d.t - 1 - w - 1; set = true; }
    if (!set) continue;
    // Source cells lie strictly inside the written ring, so the in-place
    // update does not depend on the visiting order.  An axis of one cell (a
    // coarse level of a short grid) has none: its cell stays.
    const idx_t src = d.index(max(si, 0), max(sj, 0), max(sk, 0), max(sl, 0));
    if (nc == 4) ((float4 *)a)[q] = ((const float4 *)a)[src];
    else a[q] = a[src];
  }
}
void launch_set_bound_neumann(float *a, Dims4 d, int nc, int w, cudaStream_t s) {
  BoxDecoder bx = make_decoder(d.x, d.y, d.z, 0, 0, 0, 0);
  k_set_bound_neumann<<<grid_for(d.cells(), NT), NT, 0, s>>>(a, d, bx, nc, w);
}

__global__ void k_reset_outside(float4 *a, Dims4 d, BoxDecoder bx, int rb) {
  const uint32_t n = (uint32_t)d.cells();
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < n;
       q += gridDim.x * blockDim.x) {
    int i, j, k, l;
    bx.decode(q, i, j, k, l);
    if (in_bounds(d, i, j, k, l, rb)) continue;
    a[q] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
}
void launch_reset_outside(float4 *a, Dims4 d, int resetBnd, cudaStream_t s) {
  BoxDecoder bx = make_decoder(d.x, d.y, d.z, 0, 0, 0, 0);
  k_reset_outside<<<grid_for(d.cells(), NT), NT, 0, s>>>(a, d, bx, resetBnd);
}

// ---------------------------------------------------------------------------
// Reductions (grid4d.cpp:142-172, :263-285)
// ---------------------------------------------------------------------------

__device__ __forceinline__ void post_value(const HostPost &post, float v) {
  if (!post.hr) return;
  post.hr->value = v;
  __threadfence_system();
  *(volatile unsigned int *)&post.hr->seq = post.seq;
}

template <int WHICH>
__global__ void k_reduce_minmax(const float *__restrict__ a, long long n, int nc,
                                float *partials, unsigned int *counter,
                                float *result, HostPost post) {
  __shared__ float sh[NT / 32];
  float acc = WHICH == 0 ? -FLT_MAX : FLT_MAX;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    float v;
    if (nc == 4) {
      const float4 x = __ldg((const float4 *)a + i);
      v = x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w;  // normSquare
    } else {
      v = __ldg(a + i);
    }
    if (WHICH == 0) { if (v > acc) acc = v; }
    else { if (v < acc) acc = v; }
  }
  float b = WHICH == 0 ? block_max<NT>(acc, sh) : block_min<NT>(acc, sh);
  if (threadIdx.x == 0) partials[blockIdx.x] = b;
  if (last_block_arrives(counter)) {
    float m = WHICH == 0 ? -FLT_MAX : FLT_MAX;
    for (int q = threadIdx.x; q < (int)gridDim.x; q += blockDim.x) {
      float v = __ldcg(partials + q);
      if (WHICH == 0) { if (v > m) m = v; }
      else { if (v < m) m = v; }
    }
    m = WHICH == 0 ? block_max<NT>(m, sh) : block_min<NT>(m, sh);
    if (threadIdx.x == 0) {
      *result = m;
      *counter = 0;
      post_value(post, m);
    }
  }
}
void launch_reduce_minmax(const float *a, long long ncell, int nc, int which,
                          float *partials, unsigned int *counter, float *result,
                          cudaStream_t s, HostPost post) {
  const int nb = grid_for(ncell, NT, 4);
  if (which == 0)
    k_reduce_minmax<0><<<nb, NT, 0, s>>>(a, ncell, nc, partials, counter, result, post);
  else
    k_reduce_minmax<1><<<nb, NT, 0, s>>>(a, ncell, nc, partials, counter, result, post);
}

// out = ((base + t[0]) + t[1]) + ..., each add rounded on its own, in one pass;
// with `result`, max |out|^2 as k_reduce_minmax<0> forms it.  out may be base.
struct VecTerms {
  const float4 *t[VEC_SUM_MAX];
};
__global__ void __launch_bounds__(NT)
k_vec_sum(float4 *out, const float4 *base, VecTerms terms, int nt, long long n, float *partials,
          unsigned int *counter, float *result) {
  __shared__ float sh[NT / 32];
  float acc = -FLT_MAX;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    float4 v = base[i];
    for (int k = 0; k < nt; ++k) {
      const float4 y = __ldg(terms.t[k] + i);
      v.x += y.x;
      v.y += y.y;
      v.z += y.z;
      v.w += y.w;
    }
    out[i] = v;
    const float m = v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;  // normSquare
    if (m > acc) acc = m;
  }
  if (!result) return;
  const float b = block_max<NT>(acc, sh);
  if (threadIdx.x == 0) partials[blockIdx.x] = b;
  if (last_block_arrives(counter)) {
    float m = -FLT_MAX;
    for (int q = threadIdx.x; q < (int)gridDim.x; q += blockDim.x) {
      const float v = __ldcg(partials + q);
      if (v > m) m = v;
    }
    m = block_max<NT>(m, sh);
    if (threadIdx.x == 0) {
      *result = m;
      *counter = 0;
    }
  }
}
void launch_vec_sum(float4 *out, const float4 *base, const float4 *const *terms, int nt,
                    long long ncell, float *partials, unsigned int *counter, float *result,
                    cudaStream_t s) {
  VecTerms v;
  for (int k = 0; k < VEC_SUM_MAX; ++k) v.t[k] = k < nt ? terms[k] : nullptr;
  k_vec_sum<<<grid_for(ncell, NT), NT, 0, s>>>(out, base, v, nt, ncell, partials, counter, result);
}

// calcLsDiffTempl (optflow4d.cpp:895-927).  Four cells per trip, all loads
// first: a small grid then needs a quarter of the blocks, whose partials the
// last block sums, and still has its loads in flight together.
constexpr int LSD_CPT = 4;
__global__ void __launch_bounds__(NT)
k_ls_diff(const float *__restrict__ i0, const float *__restrict__ i1, float *out, Dims4 d,
          BoxDecoder bx, uint32_t nbox, float correction, double scale, double *partials,
          unsigned int *counter, double *result_d, float *result_f, HostPost post) {
  __shared__ double sh[NT / 32];
  double acc = 0.0;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < nbox; q += LSD_CPT * stride) {
    idx_t id[LSD_CPT];
    float a[LSD_CPT], b[LSD_CPT];
    // nbox + 3 stride stays far below 2^32
#pragma unroll
    for (int m = 0; m < LSD_CPT; ++m) {
      const uint32_t n = q + m * stride;
      id[m] = -1;
      a[m] = b[m] = 0.f;  // equal signs: no contribution
      if (n < nbox) {
        int i, j, k, l;
        bx.decode(n, i, j, k, l);
        id[m] = d.index(i, j, k, l);
        a[m] = __ldg(i0 + id[m]);
        b[m] = __ldg(i1 + id[m]);
      }
    }
#pragma unroll
    for (int m = 0; m < LSD_CPT; ++m) {
      if ((a[m] < 0.f && b[m] < 0.f) || (a[m] >= 0.f && b[m] >= 0.f)) {
        if (out && id[m] >= 0) out[id[m]] = 0.f;
      } else {
        float dd = fabsf(a[m] - b[m]) * correction;
        if (dd > 1.f) dd = 1.f;
        acc += (double)dd;
        if (out) out[id[m]] = dd;
      }
    }
  }
  double b = block_sum<NT>(acc, sh);
  if (threadIdx.x == 0) partials[blockIdx.x] = b;
  if (last_block_arrives(counter)) {
    double m = 0.0;
    for (int q = threadIdx.x; q < (int)gridDim.x; q += blockDim.x) m += __ldcg(partials + q);
    m = block_sum<NT>(m, sh);
    if (threadIdx.x == 0) {
      double accu = m * 1000.;
      if (d.t > 1) accu *= 1000.;
      accu *= scale;
      *result_d = accu;
      *result_f = (float)accu;
      *counter = 0;
      post_value(post, (float)accu);
    }
  }
}
int ls_diff_blocks(Dims4 d, int bnd) {
  const long long ex = d.x - 2 * bnd, ey = d.y - 2 * bnd, ez = d.z - 2 * bnd, et = d.t - 2 * bnd;
  const long long nb = (ex > 0 && ey > 0 && ez > 0 && et > 0) ? ex * ey * ez * et : 1;
  return grid_for((nb + LSD_CPT - 1) / LSD_CPT, NT, 4);
}
void launch_ls_diff(const float *i0, const float *i1, float *out, Dims4 d,
                    float correction, int bnd, double *partials,
                    unsigned int *counter, double *result_d, float *result_f,
                    cudaStream_t s, HostPost post) {
  const int ex = d.x - 2 * bnd, ey = d.y - 2 * bnd, ez = d.z - 2 * bnd, et = d.t - 2 * bnd;
  long long nbox = (ex > 0 && ey > 0 && ez > 0 && et > 0) ? (long long)ex * ey * ez * et : 0;
  BoxDecoder bx = make_decoder(ex > 0 ? ex : 1, ey > 0 ? ey : 1, ez > 0 ? ez : 1, bnd, bnd, bnd, bnd);
  // accu *= 1. / double(sx*sy*sz*st) with int arithmetic for the count.
  // Grid4d's is3D() and is4D() are constant true (grid4d.h:82-83), so
  // FOR_IJKT_BND (kernel.h:62-68) and this count shrink every axis, T == 1
  // included.  When bnd leaves no cells the loop adds nothing and the
  // reference returns 0 * (1 / cnt): -0 for a negative count, NaN for 0.
  const int cnt = ex * ey * ez * et;
  const double scale = 1. / (double)cnt;
  k_ls_diff<<<ls_diff_blocks(d, bnd), NT, 0, s>>>(i0, i1, out, d, bx, (uint32_t)nbox,
                                                  correction, scale, partials, counter,
                                                  result_d, result_f, post);
}

// ---------------------------------------------------------------------------
// Resampling: knInterpol4d / KnInterpolateGrid4dTempl (grid4d.cpp:531-538,
// grid4d.h:463-471)
// ---------------------------------------------------------------------------

// A thread owns one (x, y, z) of the target and walks tt consecutive t.
// interpol4d's sum over x, y, z is formed once per source t plane and kept
// for the targets that share it (two of three planes when refining by two),
// so a refined cell costs 4 corner loads instead of 16.  The target positions
// depend on the indices alone, so every lane keeps and drops planes together.
// Prolonging 31x33x29x32 Vec4 by two takes 64 us against 188 us for 16 loads
// per cell (the floor of its bytes is 38 us); 8 planes a thread took 78, 32 took 70.
constexpr int RS_TT = 16;
// planes a thread: as many as still give every SM 2048 threads (a small grid is
// bound by latency: 6.9 us with one plane a thread, 22 us with 16)
static int planes_per_thread(long long cells, int most) {
  const long long n = cells / ((long long)sm_count() * 2048);
  return n < 1 ? 1 : n > most ? most : (int)n;
}
template <int NC>
__global__ void __launch_bounds__(NT, 6)
k_resample(float *__restrict__ target, Dims4 td, BoxDecoder bx, uint32_t n, int tt,
           const float *__restrict__ source, Dims4 sd, float4 fac, float4 off, float mul) {
  const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  int i, j, k, tc;
  bx.decode(q, i, j, k, tc);
  const AxisW ax = axis_index((float)i * fac.x + off.x, sd.x);
  const AxisW ay = axis_index((float)j * fac.y + off.y, sd.y);
  const AxisW az = axis_index((float)k * fac.z + off.z, sd.z);
  const int l0 = tc * tt, l1 = min(l0 + tt, td.t);
  idx_t id = td.index(i, j, k, l0);
  const idx_t sT = td.st();
  int have = -2;  // the plane sums a, b belong to source planes have, have + 1
  if (NC == 4) {
    const float4 *src = (const float4 *)source;
    const Corner c = corner_of(sd, ax.b, ay.b, az.b, 0);
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
    for (int l = l0; l < l1; ++l, id += sT) {
      const AxisW at = axis_index((float)l * fac.w + off.w, sd.t);
      if (at.b != have) {
        const uint32_t p = c.i + (uint32_t)c.sT * (uint32_t)at.b;
        a = at.b == have + 1 ? b : plane_vec(src, c, p, ax, ay, az);
        b = plane_vec(src, c, p + (uint32_t)c.sT, ax, ay, az);
        have = at.b;
      }
      float4 v = weigh2(a, b, at);
      if (mul != 1.f) v = make_float4(v.x * mul, v.y * mul, v.z * mul, v.w * mul);
      ((float4 *)target)[id] = v;
    }
  } else {
    const Corner c = corner_of(sd, ax.b, ay.b, az.b, 0);
    float a = 0.f, b = 0.f;
    for (int l = l0; l < l1; ++l, id += sT) {
      const AxisW at = axis_index((float)l * fac.w + off.w, sd.t);
      if (at.b != have) {
        const uint32_t p = c.i + (uint32_t)c.sT * (uint32_t)at.b;
        a = at.b == have + 1 ? b : plane_real(source, c, p, ax, ay, az);
        b = plane_real(source, c, p + (uint32_t)c.sT, ax, ay, az);
        have = at.b;
      }
      const float v = a * at.w0 + b * at.w1;
      target[id] = mul != 1.f ? v * mul : v;
    }
  }
}
// One cell per thread, all its corner loads at once: for targets that share no
// source plane sums.  Through the walk these took up to a third longer: 40 x 38
// x 41 x 32 restricted by two 6.8 -> 6.1 us, 56^3 x 40 9.8 -> 8.1, 12^4 refined by
// 3/2 8.1 -> 6.1, 48^4 Vec4 restricted 12.2 -> 10.9.
template <int NC>
__global__ void __launch_bounds__(NT)
k_resample_one(float *__restrict__ target, Dims4 td, BoxDecoder bx, uint32_t n,
               const float *__restrict__ source, Dims4 sd, float4 fac, float4 off, float mul) {
  const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  int i, j, k, l;
  bx.decode(q, i, j, k, l);
  const AxisW ax = axis_index((float)i * fac.x + off.x, sd.x);
  const AxisW ay = axis_index((float)j * fac.y + off.y, sd.y);
  const AxisW az = axis_index((float)k * fac.z + off.z, sd.z);
  const AxisW at = axis_index((float)l * fac.w + off.w, sd.t);
  const Corner c = corner_of(sd, ax.b, ay.b, az.b, 0);
  const uint32_t p = c.i + (uint32_t)c.sT * (uint32_t)at.b;
  if (NC == 4) {
    const float4 *src = (const float4 *)source;
    const float4 a = plane_vec(src, c, p, ax, ay, az);
    const float4 b = plane_vec(src, c, p + (uint32_t)c.sT, ax, ay, az);
    float4 v = weigh2(a, b, at);
    if (mul != 1.f) v = make_float4(v.x * mul, v.y * mul, v.z * mul, v.w * mul);
    ((float4 *)target)[q] = v;
  } else {
    const float a = plane_real(source, c, p, ax, ay, az);
    const float b = plane_real(source, c, p + (uint32_t)c.sT, ax, ay, az);
    const float v = a * at.w0 + b * at.w1;
    target[q] = mul != 1.f ? v * mul : v;
  }
}
// A source with an axis of one cell, as the coarse levels of a short grid have
// (24^3 x 3 halves to 12^3 x 1).  Such an axis has no second corner: every
// position takes its cell with weight 1, and the stride 0 keeps the corner
// of weight 0 inside the grid (the kernels above would read a plane before it).
struct ThinAxis {
  AxisW w;
  idx_t step;
};
__device__ __forceinline__ ThinAxis thin_axis(float p, int n, idx_t stride) {
  if (n < 2) return ThinAxis{AxisW{0, 1.f, 0.f}, 0};
  return ThinAxis{axis_index(p, n), stride};
}
__global__ void __launch_bounds__(NT)
k_resample_thin(float *__restrict__ target, Dims4 td, BoxDecoder bx, uint32_t n,
                const float *__restrict__ source, Dims4 sd, int nc, float4 fac, float4 off,
                float mul) {
  const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  int i, j, k, l;
  bx.decode(q, i, j, k, l);
  const ThinAxis x = thin_axis((float)i * fac.x + off.x, sd.x, nc);
  const ThinAxis y = thin_axis((float)j * fac.y + off.y, sd.y, (idx_t)sd.x * nc);
  const ThinAxis z = thin_axis((float)k * fac.z + off.z, sd.z, sd.sz() * nc);
  const ThinAxis t = thin_axis((float)l * fac.w + off.w, sd.t, sd.st() * nc);
  const float *base = source + sd.index(x.w.b, y.w.b, z.w.b, t.w.b) * nc;
  for (int c = 0; c < nc; ++c) {
    float plane[2];
    for (int m = 0; m < 2; ++m) {
      const float *p = base + c + m * t.step, *py = p + y.step, *pz = p + z.step, *pyz = py + z.step;
      plane[m] = plane_sum(__ldg(p), __ldg(py), __ldg(p + x.step), __ldg(py + x.step), __ldg(pz),
                           __ldg(pyz), __ldg(pz + x.step), __ldg(pyz + x.step), x.w, y.w, z.w);
    }
    const float v = plane[0] * t.w.w0 + plane[1] * t.w.w1;
    target[(size_t)q * nc + c] = mul != 1.f ? v * mul : v;
  }
}
void launch_resample(float *target, Dims4 td, const float *source, Dims4 sd,
                     int nc, float4 fac, float4 off, cudaStream_t s, float mul) {
  if (td.cells() <= 0) return;
  BoxDecoder bx = make_decoder(td.x, td.y, td.z, 0, 0, 0, 0);
  if (sd.x < 2 || sd.y < 2 || sd.z < 2 || sd.t < 2) {
    const uint32_t n = (uint32_t)td.cells();
    k_resample_thin<<<grid_all(n), NT, 0, s>>>(target, td, bx, n, source, sd, nc, fac, off, mul);
    return;
  }
  const int tt = planes_per_thread(td.cells(), RS_TT);
  // a thread with one plane has nothing to keep, and targets two source planes
  // apart (restriction by two) share none
  if (tt == 1 || fac.w >= 2.f) {
    const uint32_t n = (uint32_t)td.cells();
    if (nc == 4)
      k_resample_one<4><<<grid_all(n), NT, 0, s>>>(target, td, bx, n, source, sd, fac, off, mul);
    else
      k_resample_one<1><<<grid_all(n), NT, 0, s>>>(target, td, bx, n, source, sd, fac, off, mul);
    return;
  }
  const uint32_t n = (uint32_t)(td.st() * ((td.t + tt - 1) / tt));
  if (nc == 4)
    k_resample<4><<<grid_all(n), NT, 0, s>>>(target, td, bx, n, tt, source, sd, fac, off, mul);
  else
    k_resample<1><<<grid_all(n), NT, 0, s>>>(target, td, bx, n, tt, source, sd, fac, off, mul);
}

// ---------------------------------------------------------------------------
// semiLagrange4d (optflow4d.cpp:1275-1290): dst = src(ijkt+0.5 - vel*dt) over
// bnd=1 cells of a fresh (zeroed) grid.
// ---------------------------------------------------------------------------

// With `maxn2` set, the launch is the single substep of advectCflHelper4d
// (optflow4d.cpp:1309-1321): the substep count int(maxVel/cfl)+1 is
// evaluated here from the device-resident max |v|^2, and a count other than
// one is reported through `flag` so that the host can redo the call with
// host-side substeps.
template <int NC>
__global__ void __launch_bounds__(NT)
k_advect(const float4 *__restrict__ vel, const float *__restrict__ src, float *__restrict__ dst,
         Dims4 d, BoxDecoder bx, float dt, const float *maxn2, float cfl, int *flag) {
  if (maxn2 && blockIdx.x == 0 && threadIdx.x == 0) {
    const float maxVel = sqrtf(*maxn2) * 1.0f;
    const int steps = trunc_i(maxVel / cfl) + 1;
    if (steps != 1) *flag = 1;
  }
  const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= (uint32_t)d.cells()) return;
  int i, j, k, l;
  bx.decode(q, i, j, k, l);
  if (!in_bounds(d, i, j, k, l, 1)) {
    if (NC == 4) ((float4 *)dst)[q] = make_float4(0.f, 0.f, 0.f, 0.f);
    else dst[q] = 0.f;
    return;
  }
  const float4 v = __ldg(vel + q);
  const float p0 = (float)(i + 0.5f) - v.x * dt;
  const float p1 = (float)(j + 0.5f) - v.y * dt;
  const float p2 = (float)(k + 0.5f) - v.z * dt;
  const float p3 = (float)(l + 0.5f) - v.w * dt;
  if (NC == 4)
    ((float4 *)dst)[q] = interp4_vec((const float4 *)src, d, p0, p1, p2, p3);
  else
    dst[q] = interp4_real(src, d, p0, p1, p2, p3);
}
static void advect_any(const float4 *vel, const float *src, float *dst, Dims4 d, int nc, float dt,
                       const float *maxn2, float cfl, int *flag, cudaStream_t s) {
  BoxDecoder bx = make_decoder(d.x, d.y, d.z, 0, 0, 0, 0);
  const unsigned nb = grid_all(d.cells());
  if (nc == 4)
    k_advect<4><<<nb, NT, 0, s>>>(vel, src, dst, d, bx, dt, maxn2, cfl, flag);
  else
    k_advect<1><<<nb, NT, 0, s>>>(vel, src, dst, d, bx, dt, maxn2, cfl, flag);
}
void launch_advect(const float4 *vel, const float *src, float *dst, Dims4 d,
                   int nc, float dt, cudaStream_t s) {
  advect_any(vel, src, dst, d, nc, dt, nullptr, 0.f, nullptr, s);
}

void launch_advect_cfl1(const float4 *vel, const float *src, float *dst, Dims4 d, int nc,
                        const float *maxn2, float cfl, int *flag, cudaStream_t s) {
  advect_any(vel, src, dst, d, nc, (1.0f / (float)1) * 1.0f, maxn2, cfl, flag, s);
}

// The driver's warp in one pass: dst = the single-substep advection of src
// (k_advect with maxn2), setBoundNeumann(0) of it, and calcLsDiff4d of the
// result against i1 over the bnd box.  A cell of the outermost ring takes the
// value of its source cell, which lies inside it (every extent at least 3), by
// advecting that cell itself: the same operations, so the same bits as copying
// it afterwards.  One pass instead of four over the
// grid and, for a small level, one launch instead of four.
__global__ void __launch_bounds__(NT)
k_warp_error(const float4 *__restrict__ vel, const float *__restrict__ src, float *__restrict__ dst,
             const float *__restrict__ i1, Dims4 d, BoxDecoder bx, const float *maxn2, float cfl,
             int *flag, float correction, int bnd, double scale, double *partials,
             unsigned int *counter, double *result_d, float *result_f, HostPost post) {
  __shared__ double sh[NT / 32];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const float maxVel = sqrtf(*maxn2) * 1.0f;
    const int steps = trunc_i(maxVel / cfl) + 1;
    if (steps != 1) *flag = 1;
  }
  double acc = 0.0;
  const uint32_t n = (uint32_t)d.cells();
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    int c[4];
    bx.decode(q, c[0], c[1], c[2], c[3]);
    const bool box = in_bounds(d, c[0], c[1], c[2], c[3], bnd);
    const int ext[4] = {d.x, d.y, d.z, d.t};
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int o = c[a];
      if (o <= 0) c[a] = 1;
      if (o >= ext[a] - 1) c[a] = ext[a] - 2;
    }
    const float4 v = __ldg(vel + d.index(c[0], c[1], c[2], c[3]));
    const float dt = 1.0f;
    const float w = interp4_real(src, d, (float)(c[0] + 0.5f) - v.x * dt,
                                 (float)(c[1] + 0.5f) - v.y * dt, (float)(c[2] + 0.5f) - v.z * dt,
                                 (float)(c[3] + 0.5f) - v.w * dt);
    dst[q] = w;
    if (box) {
      const float b = __ldg(i1 + q);
      if (!((w < 0.f && b < 0.f) || (w >= 0.f && b >= 0.f))) {
        float dd = fabsf(w - b) * correction;
        if (dd > 1.f) dd = 1.f;
        acc += (double)dd;
      }
    }
  }
  double b = block_sum<NT>(acc, sh);
  if (threadIdx.x == 0) partials[blockIdx.x] = b;
  if (last_block_arrives(counter)) {
    double m = 0.0;
    for (int q = threadIdx.x; q < (int)gridDim.x; q += blockDim.x) m += __ldcg(partials + q);
    m = block_sum<NT>(m, sh);
    if (threadIdx.x == 0) {
      double accu = m * 1000.;
      if (d.t > 1) accu *= 1000.;
      accu *= scale;
      *result_d = accu;
      *result_f = (float)accu;
      *counter = 0;
      post_value(post, (float)accu);
    }
  }
}
bool launch_warp_error(const float4 *vel, const float *src, float *dst, const float *i1, Dims4 d,
                       const float *maxn2, float cfl, int *flag, float correction, int bnd,
                       double *partials, unsigned int *counter, double *result_d, float *result_f,
                       cudaStream_t s, HostPost post) {
  if (d.x < 3 || d.y < 3 || d.z < 3 || d.t < 3) return false;
  static const int per_sm = [] {
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_warp_error, NT, 0);
    return n < 1 ? 1 : n;
  }();
  const int ex = d.x - 2 * bnd, ey = d.y - 2 * bnd, ez = d.z - 2 * bnd, et = d.t - 2 * bnd;
  const int cnt = ex * ey * ez * et;  // as launch_ls_diff
  k_warp_error<<<grid_for(d.cells(), NT, per_sm), NT, 0, s>>>(
      vel, src, dst, i1, d, make_decoder(d.x, d.y, d.z, 0, 0, 0, 0), maxn2, cfl, flag, correction,
      bnd, 1. / (double)cnt, partials, counter, result_d, result_f, post);
  return true;
}

// Bound by instruction issue (about 330 per cell, most of them index and
// address arithmetic of the 32 corner loads): 64^4 in 183 us, 302 us with
// 64-bit indices and a capped grid; the floor of its bytes is 110 us.
__global__ void __launch_bounds__(NT, 8)
k_deform_twoway(const float4 *__restrict__ vel, const float4 *__restrict__ velInv,
                const float *__restrict__ i0, const float *__restrict__ i1,
                float *__restrict__ out, Dims4 d, BoxDecoder bx, float alpha, float alphaInv) {
  const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= (uint32_t)d.cells()) return;
  int i, j, k, l;
  bx.decode(q, i, j, k, l);
  float a0 = 0.f, a1 = 0.f;
  if (in_bounds(d, i, j, k, l, 1)) {
    const float4 v = __ldg(vel + q);
    const float4 w = __ldg(velInv + q);
    a0 = interp4_real(i0, d, (float)(i + 0.5f) - v.x * alpha, (float)(j + 0.5f) - v.y * alpha,
                           (float)(k + 0.5f) - v.z * alpha, (float)(l + 0.5f) - v.w * alpha);
    a1 = interp4_real(i1, d, (float)(i + 0.5f) - w.x * alphaInv,
                           (float)(j + 0.5f) - w.y * alphaInv, (float)(k + 0.5f) - w.z * alphaInv,
                           (float)(l + 0.5f) - w.w * alphaInv);
  }
  out[q] = a0 * alphaInv + alpha * a1;
}
void launch_deform_twoway(const float4 *vel, const float4 *velInv,
                          const float *i0, const float *i1, float *out, Dims4 d,
                          float alpha, float alphaInv, cudaStream_t s) {
  BoxDecoder bx = make_decoder(d.x, d.y, d.z, 0, 0, 0, 0);
  k_deform_twoway<<<grid_all(d.cells()), NT, 0, s>>>(vel, velInv, i0, i1, out, d, bx, alpha,
                                                     alphaInv);
}

// ---------------------------------------------------------------------------
// Mode-3 hi-res slice lookup (optflow4d.cpp:1648-1665, :2009-2013)
// ---------------------------------------------------------------------------

__global__ void k_blend_slices(const float4 *__restrict__ v1, const float4 *__restrict__ v2,
                               float4 *__restrict__ vt, long long n, float f1, float f2) {
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
       q += (long long)gridDim.x * blockDim.x) {
    const float4 a = __ldg(v1 + q), b = __ldg(v2 + q);
    float4 r;
    r.x = 0.f + f1 * a.x; r.x += f2 * b.x;
    r.y = 0.f + f1 * a.y; r.y += f2 * b.y;
    r.z = 0.f + f1 * a.z; r.z += f2 * b.z;
    r.w = 0.f + f1 * a.w; r.w += f2 * b.w;
    vt[q] = r;
  }
}
void launch_blend_slices(const float4 *v1, const float4 *v2, float4 *vt,
                         long long cells, float f1, float f2, cudaStream_t s) {
  k_blend_slices<<<grid_for(cells, NT), NT, 0, s>>>(v1, v2, vt, cells, f1, f2);
}

// The blends of both directions of a two-way frame in one launch: cells of
// the first set, then of the second, each blended as k_blend_slices does.
struct BlendSet {
  const float4 *v1, *v2;
  float4 *vt;
  float f1, f2;
};
__global__ void k_blend_slices2(BlendSet a, BlendSet b, long long n) {
  pdl_wait();
  pdl_launch_dependents();
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < 2 * n;
       q += (long long)gridDim.x * blockDim.x) {
    const BlendSet &S = q < n ? a : b;
    const long long e = q < n ? q : q - n;
    const float4 x = __ldg(S.v1 + e), y = __ldg(S.v2 + e);
    float4 r;
    r.x = 0.f + S.f1 * x.x; r.x += S.f2 * y.x;
    r.y = 0.f + S.f1 * x.y; r.y += S.f2 * y.y;
    r.z = 0.f + S.f1 * x.z; r.z += S.f2 * y.z;
    r.w = 0.f + S.f1 * x.w; r.w += S.f2 * y.w;
    S.vt[e] = r;
  }
}
void launch_blend_slices2(const float4 *v1a, const float4 *v2a, float4 *vta, float fa1, float fa2,
                          const float4 *v1b, const float4 *v2b, float4 *vtb, float fb1, float fb2,
                          long long cells, cudaStream_t s) {
  launch_pdl(k_blend_slices2, (unsigned)grid_for(2 * cells, NT), NT, s,
             BlendSet{v1a, v2a, vta, fa1, fa2}, BlendSet{v1b, v2b, vtb, fb1, fb2}, cells);
}

// interpol<Vec4> (source/util/interpol.h:57-116) of a blended slice at one
// (x, y), walking z: the sum over x and y is formed once per slice plane and
// kept for the cells that share it.
struct SliceWalk {
  const float4 *base;  // the (x, y) corner in z plane 0
  AxisW ax, ay;
  idx_t sY, sZ;
  int have;
  float4 a, b;  // planes have, have + 1
  __device__ __forceinline__ void init(const float4 *vt, int vx, int vy, const AxisW &wx,
                                       const AxisW &wy) {
    ax = wx;
    ay = wy;
    sY = vx;
    sZ = (idx_t)vx * vy;
    base = vt + ((uint32_t)wx.b + (uint32_t)vx * (uint32_t)wy.b);
    have = -2;
    a = b = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __device__ __forceinline__ float4 plane(const float4 *p) const {
    const float4 c0 = __ldg(p), c1 = __ldg(p + sY), c2 = __ldg(p + 1), c3 = __ldg(p + sY + 1);
    return make_float4((c0.x * ay.w0 + c1.x * ay.w1) * ax.w0 + (c2.x * ay.w0 + c3.x * ay.w1) * ax.w1,
                       (c0.y * ay.w0 + c1.y * ay.w1) * ax.w0 + (c2.y * ay.w0 + c3.y * ay.w1) * ax.w1,
                       (c0.z * ay.w0 + c1.z * ay.w1) * ax.w0 + (c2.z * ay.w0 + c3.z * ay.w1) * ax.w1,
                       (c0.w * ay.w0 + c1.w * ay.w1) * ax.w0 + (c2.w * ay.w0 + c3.w * ay.w1) * ax.w1);
  }
  __device__ __forceinline__ float4 at(const AxisW &az) {
    if (az.b != have) {
      const float4 *p = base + sZ * az.b;
      a = az.b == have + 1 ? b : plane(p);
      b = plane(p + sZ);
      have = az.b;
    }
    return weigh2(a, b, az);
  }
};

// A thread owns one (x, y) of the frame and zn <= LK_Z consecutive z.  TWO: both
// directions and their blend, dst.multConst(1-alpha); dst.addScaled(dst1,
// alpha).  Bound by instruction issue and the gathers' latency: a 128^3 frame
// two-way with its blend takes 30 us against 33 us for a trilinear sample per
// cell; 2, 4, 6 or 8 cells a thread, or 4 blocks per SM, were slower.
constexpr int LK_Z = 3;
template <bool TWO>
__global__ void __launch_bounds__(NT, 5)
k_lookup_slice(float *__restrict__ dst, int dx, int dy, BoxDecoder bx, uint32_t n, int zend, int zn,
               const float *__restrict__ phi0, const float *__restrict__ phi1, Dims4 pd,
               float time, float dt0, float dt1, const float4 *__restrict__ vt0,
               const float4 *__restrict__ vt1, int vx, int vy, int vz, float4 sf3, float4 off3,
               float4 df) {
  pdl_wait();
  const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  int i, j, kc, unused;
  bx.decode(q, i, j, kc, unused);
  const AxisW ax = axis_index((float)i * sf3.x + off3.x, vx);
  const AxisW ay = axis_index((float)j * sf3.y + off3.y, vy);
  // bx.oz is the first z of the box, kc the chunk plus it
  const int k0 = bx.oz + (kc - bx.oz) * zn;
  float r[LK_Z];
  // one direction after the other: only one slice's planes are then held in
  // registers (75 registers and three blocks per SM with both)
  auto walk = [&](const float *phi, const float4 *vt, float dt, auto &&use) {
    SliceWalk w;
    w.init(vt, vx, vy, ax, ay);
#pragma unroll
    for (int m = 0; m < LK_Z; ++m) {
      const int k = k0 + m;
      if (m >= zn || k >= zend) break;
      float4 v = w.at(axis_index((float)k * sf3.z + off3.z, vz));
      v.x *= df.x;
      v.y *= df.y;
      v.z *= df.z;
      v.w *= df.w;
      use(m, interp4_real(phi, pd, (float)(i + 0.5f) - v.x * dt, (float)(j + 0.5f) - v.y * dt,
                               (float)(k + 0.5f) - v.z * dt, (time + 0.5f) - v.w * dt));
    }
  };
  const idx_t id = (idx_t)i + (idx_t)dx * j, sZ = (idx_t)dx * dy;
  if (TWO) {
    walk(phi0, vt0, dt0, [&](int m, float a) { r[m] = a * dt1; });
    walk(phi1, vt1, dt1, [&](int m, float b) { dst[id + sZ * (k0 + m)] = r[m] + dt0 * b; });
  } else {
    walk(phi0, vt0, dt0, [&](int m, float a) { dst[id + sZ * (k0 + m)] = a; });
  }
}

static void lookup_box(int dx, int dy, int dz, int bordSkip, int &lo, int &ex,
                       int &ey, int &ez, int minBnd = 10) {
  lo = bordSkip > minBnd ? bordSkip : minBnd;
  ex = dx - 2 * lo;
  ey = dy - 2 * lo;
  ez = dz - 2 * lo;
}

template <bool TWO>
static void lookup_launch(float *dst, int dx, int dy, int dz, const float *phi0, const float *phi1,
                          Dims4 pd, float time, float dt0, float dt1, const float4 *vt0,
                          const float4 *vt1, int vx, int vy, int vz, float4 sf3, float4 off3,
                          float4 df, int bordSkip, int minBnd, cudaStream_t s) {
  int lo, ex, ey, ez;
  lookup_box(dx, dy, dz, bordSkip, lo, ex, ey, ez, minBnd);
  if (ex <= 0 || ey <= 0 || ez <= 0) return;
  const int zn = planes_per_thread((long long)ex * ey * ez, LK_Z), zc = (ez + zn - 1) / zn;
  BoxDecoder bx = make_decoder(ex, ey, zc, lo, lo, lo, 0);
  const uint32_t n = (uint32_t)((long long)ex * ey * zc);
  launch_pdl(k_lookup_slice<TWO>, grid_all(n), NT, s, dst, dx, dy, bx, n, lo + ez, zn, phi0, phi1,
             pd, time, dt0, dt1, vt0, vt1, vx, vy, vz, sf3, off3, df);
}

void launch_lookup_slice(float *dst, int dx, int dy, int dz, const float *phi,
                         Dims4 pd, float time, float dt, const float4 *vt,
                         int vx, int vy, int vz, float4 sf3, float4 off3,
                         float4 defoFactor, int bordSkip, cudaStream_t s, int minBnd) {
  lookup_launch<false>(dst, dx, dy, dz, phi, phi, pd, time, dt, 0.f, vt, vt, vx, vy, vz, sf3, off3,
                       defoFactor, bordSkip, minBnd, s);
}
void launch_lookup_slice_twoway(float *dst, int dx, int dy, int dz,
                                const float *phi0, const float *phi1, Dims4 pd,
                                float time, float alpha, float alphaInv,
                                const float4 *vt0, const float4 *vt1, int vx,
                                int vy, int vz, float4 sf3, float4 off3,
                                float4 defoFactor, int bordSkip, cudaStream_t s) {
  lookup_launch<true>(dst, dx, dy, dz, phi0, phi1, pd, time, alpha, alphaInv, vt0, vt1, vx, vy, vz,
                      sf3, off3, defoFactor, bordSkip, 10, s);
}

}  // namespace flof
