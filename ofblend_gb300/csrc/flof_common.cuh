// flof_common.cuh -- device-side building blocks shared by the FlOF kernels.
//
// Layout (reference source/grid4d.h:92-97): a 4D grid (X,Y,Z,T) is stored
// x-fastest, idx = i + X*j + X*Y*k + X*Y*Z*t.  Real grids are float, Vec4
// grids are float4 (interleaved x,y,z,t), 16-byte aligned.
//
// Arithmetic: every translation unit is compiled with -fmad=false so that
// multiplies and adds are rounded separately, in the order written, like the
// reference's x86 build; fused multiply-adds appear only where a kernel asks
// for them explicitly (__fmaf_rn) and the reference has no bitwise claim.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace flof {

typedef long long idx_t;

struct Dims4 {
  int x, y, z, t;
  __host__ __device__ idx_t cells() const { return (idx_t)x * y * z * t; }
  __host__ __device__ idx_t sz() const { return (idx_t)x * y; }
  __host__ __device__ idx_t st() const { return (idx_t)x * y * z; }
  __host__ __device__ idx_t index(int i, int j, int k, int l) const {
    return (idx_t)i + (idx_t)x * j + (idx_t)x * y * k + (idx_t)x * y * z * l;
  }
};

// Unsigned division by an invariant divisor with a multiply-high
// (Granlund & Montgomery, PLDI 1994, "round-up" variant).  Valid for every
// 32-bit dividend.
struct FastDiv {
  uint32_t d, m, l;
  FastDiv() : d(1), m(0), l(0) {}
  explicit FastDiv(uint32_t div) : d(div) {
    l = 0;
    while ((1ull << l) < div) ++l;
    uint64_t mm = ((1ull << 32) * ((1ull << l) - div)) / div + 1;
    m = (uint32_t)mm;
  }
  __device__ __forceinline__ uint32_t div(uint32_t n) const {
    uint64_t hi = __umulhi(n, m);
    return (uint32_t)((hi + n) >> l);
  }
};

// Cell coordinates of a linear index over a box of extents (ex,ey,ez,*).
struct BoxDecoder {
  FastDiv fx, fy, fz;
  int ox, oy, oz, ot;  // coordinate offsets added after decoding
  uint32_t ex, ey, ez;
  __device__ __forceinline__ void decode(uint32_t n, int &i, int &j, int &k,
                                         int &l) const {
    uint32_t q = fx.div(n);
    i = (int)(n - q * ex) + ox;
    uint32_t q2 = fy.div(q);
    j = (int)(q - q2 * ey) + oy;
    uint32_t q3 = fz.div(q2);
    k = (int)(q2 - q3 * ez) + oz;
    l = (int)q3 + ot;
  }
};

inline BoxDecoder make_decoder(int ex, int ey, int ez, int ox, int oy, int oz,
                               int ot) {
  BoxDecoder b;
  b.fx = FastDiv((uint32_t)ex);
  b.fy = FastDiv((uint32_t)ey);
  b.fz = FastDiv((uint32_t)ez);
  b.ex = (uint32_t)ex;
  b.ey = (uint32_t)ey;
  b.ez = (uint32_t)ez;
  b.ox = ox;
  b.oy = oy;
  b.oz = oz;
  b.ot = ot;
  return b;
}

__device__ __forceinline__ bool in_bounds(const Dims4 &d, int i, int j, int k,
                                          int l, int b) {
  return i >= b && j >= b && i < d.x - b && j < d.y - b && k >= b &&
         k < d.z - b && l >= b && l < d.t - b;
}

// float -> int truncation (cvt.rzi.s32.f32: NaN gives 0, out of range
// saturates); equal to the reference's (int) cast for all in-range values.
__device__ __forceinline__ int trunc_i(float p) { return __float2int_rz(p); }

// One axis of the reference's BUILD_INDEX_4D (source/util/vector4d.h:422-470;
// `1. - s1` is evaluated in double there, which for a float s1 equals
// 1.0f - s1): base index b and the weights (w0, w1) of b and
// b + 1 for a sample at p on an axis of n cells.
struct AxisW {
  int b;
  float w0, w1;
};

// n is at least 2: the corner at b + 1 is read whatever its weight.
// A position below 0 is clamped before the index is taken, which gives b = 0
// and the weights (1, 0) without three selects; NaN stays NaN (max.NaN).
__device__ __forceinline__ AxisW axis_index(float p, int n) {
  AxisW a;
  float px = p - 0.5f;
  asm("max.NaN.f32 %0, %0, 0f00000000;" : "+f"(px));
  a.b = trunc_i(px);
  a.w1 = px - (float)a.b;
  a.w0 = 1.0f - a.w1;
  if (a.b >= n - 1) { a.b = n - 2; a.w0 = 0.f; a.w1 = 1.f; }
  return a;
}

// The base corner of a quadrilinear sample: its index (grids hold fewer than
// 2^31 cells) and the strides along y, z, t.  The strides are the same for
// every thread, so a corner load is the thread's one base pointer plus uniform
// offsets: 64^4 two-way deform, 329 instructions a cell against 341 with
// 64-bit index sums and 382 with 32-bit byte offsets.
struct Corner {
  uint32_t i;
  idx_t sY, sZ, sT;
};
__device__ __forceinline__ Corner corner_of(const Dims4 &d, int bx, int by, int bz, int bt) {
  Corner c;
  c.sY = d.x;
  c.sZ = d.sz();
  c.sT = d.st();
  c.i = (uint32_t)bx +
        (uint32_t)d.x * ((uint32_t)by + (uint32_t)d.y * ((uint32_t)bz + (uint32_t)d.z * (uint32_t)bt));
  return c;
}
// interpol4d's sum (vector4d.h:497-512) over one t plane, pairs along y, then
// x and z; the planes at t and t + 1 are then weighted and added.
__device__ __forceinline__ float plane_sum(float c0, float c1, float c2, float c3, float c4,
                                           float c5, float c6, float c7, const AxisW &ax,
                                           const AxisW &ay, const AxisW &az) {
  return ((c0 * ay.w0 + c1 * ay.w1) * ax.w0 + (c2 * ay.w0 + c3 * ay.w1) * ax.w1) * az.w0 +
         ((c4 * ay.w0 + c5 * ay.w1) * ax.w0 + (c6 * ay.w0 + c7 * ay.w1) * ax.w1) * az.w1;
}
// the plane whose base corner is p[i]
__device__ __forceinline__ float plane_real(const float *__restrict__ p, const Corner &c,
                                            uint32_t i, const AxisW &ax, const AxisW &ay,
                                            const AxisW &az) {
  const float *q = p + i;
  const float *qy = q + c.sY, *qz = q + c.sZ, *qyz = q + (c.sY + c.sZ);
  return plane_sum(__ldg(q), __ldg(qy), __ldg(q + 1), __ldg(qy + 1), __ldg(qz), __ldg(qyz),
                   __ldg(qz + 1), __ldg(qyz + 1), ax, ay, az);
}
__device__ __forceinline__ float4 plane_vec(const float4 *__restrict__ p, const Corner &c,
                                            uint32_t i, const AxisW &ax, const AxisW &ay,
                                            const AxisW &az) {
  const float4 *q = p + i;
  const float4 *qy = q + c.sY, *qz = q + c.sZ, *qyz = q + (c.sY + c.sZ);
  const float4 c0 = __ldg(q), c1 = __ldg(qy), c2 = __ldg(q + 1), c3 = __ldg(qy + 1);
  const float4 c4 = __ldg(qz), c5 = __ldg(qyz), c6 = __ldg(qz + 1), c7 = __ldg(qyz + 1);
  return make_float4(
      plane_sum(c0.x, c1.x, c2.x, c3.x, c4.x, c5.x, c6.x, c7.x, ax, ay, az),
      plane_sum(c0.y, c1.y, c2.y, c3.y, c4.y, c5.y, c6.y, c7.y, ax, ay, az),
      plane_sum(c0.z, c1.z, c2.z, c3.z, c4.z, c5.z, c6.z, c7.z, ax, ay, az),
      plane_sum(c0.w, c1.w, c2.w, c3.w, c4.w, c5.w, c6.w, c7.w, ax, ay, az));
}
__device__ __forceinline__ float4 weigh2(const float4 &a, const float4 &b, const AxisW &w) {
  return make_float4(a.x * w.w0 + b.x * w.w1, a.y * w.w0 + b.y * w.w1, a.z * w.w0 + b.z * w.w1,
                     a.w * w.w0 + b.w * w.w1);
}
__device__ __forceinline__ float interp4_real(const float *__restrict__ data, const Dims4 &d,
                                              float p0, float p1, float p2, float p3) {
  const AxisW ax = axis_index(p0, d.x), ay = axis_index(p1, d.y);
  const AxisW az = axis_index(p2, d.z), at = axis_index(p3, d.t);
  const Corner c = corner_of(d, ax.b, ay.b, az.b, at.b);
  const float a = plane_real(data, c, c.i, ax, ay, az);
  const float b = plane_real(data, c, c.i + (uint32_t)c.sT, ax, ay, az);
  return a * at.w0 + b * at.w1;
}
__device__ __forceinline__ float4 interp4_vec(const float4 *__restrict__ data, const Dims4 &d,
                                              float p0, float p1, float p2, float p3) {
  const AxisW ax = axis_index(p0, d.x), ay = axis_index(p1, d.y);
  const AxisW az = axis_index(p2, d.z), at = axis_index(p3, d.t);
  const Corner c = corner_of(d, ax.b, ay.b, az.b, at.b);
  const float4 a = plane_vec(data, c, c.i, ax, ay, az);
  const float4 b = plane_vec(data, c, c.i + (uint32_t)c.sT, ax, ay, az);
  return weigh2(a, b, at);
}

// interpol<Real> (source/util/interpol.h:57-95) on a 3D Real grid of extents
// size[0..2] with z stride sZ: same index build as
// axis_index, summed along y, then x and z.
__device__ __forceinline__ float interp3_real(const float *__restrict__ data, const int size[3],
                                              idx_t sZ, float q0, float q1, float q2) {
  const float px = q0 - 0.5f, py = q1 - 0.5f, pz = q2 - 0.5f;
  int xi = trunc_i(px), yi = trunc_i(py), zi = trunc_i(pz);
  float s1 = px - (float)xi, s0 = 1.0f - s1;
  float t1 = py - (float)yi, t0 = 1.0f - t1;
  float f1 = pz - (float)zi, f0 = 1.0f - f1;
  if (px < 0.f) { xi = 0; s0 = 1.f; s1 = 0.f; }
  if (py < 0.f) { yi = 0; t0 = 1.f; t1 = 0.f; }
  if (pz < 0.f) { zi = 0; f0 = 1.f; f1 = 0.f; }
  if (xi >= size[0] - 1) { xi = size[0] - 2; s0 = 0.f; s1 = 1.f; }
  if (yi >= size[1] - 1) { yi = size[1] - 2; t0 = 0.f; t1 = 1.f; }
  if (size[2] > 1) {
    if (zi >= size[2] - 1) { zi = size[2] - 2; f0 = 0.f; f1 = 1.f; }
  }
  const idx_t X = 1, Y = size[0], Z = sZ;
  const idx_t i = (idx_t)xi + Y * yi + Z * zi;
  return ((__ldg(data + i) * t0 + __ldg(data + i + Y) * t1) * s0 +
          (__ldg(data + i + X) * t0 + __ldg(data + i + X + Y) * t1) * s1) *
             f0 +
         ((__ldg(data + i + Z) * t0 + __ldg(data + i + Y + Z) * t1) * s0 +
          (__ldg(data + i + X + Z) * t0 + __ldg(data + i + X + Y + Z) * t1) * s1) *
             f1;
}

// ---- BF16 storage of Vec4 data ----------------------------------------------------

// Four bfloat16 values (x, y, z, w) in 8 bytes.  bf16 -> float is exact (the
// bf16 bits are the top half of the float); float -> bf16 rounds to nearest
// even (to_bf4).
struct __align__(8) BF4 {
  unsigned short x, y, z, w;
};
__device__ __forceinline__ float4 ld_g(const float4 *__restrict__ g, idx_t i) {
  return __ldg(g + i);
}
__device__ __forceinline__ float4 ld_g(const BF4 *__restrict__ g, idx_t i) {
  const uint2 u = __ldg((const uint2 *)(g + i));
  return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u),
                     __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
}
// The same split in two: g_raw loads the stored value, g_value widens it.
__device__ __forceinline__ float4 g_raw(const float4 *__restrict__ g, idx_t i) {
  return __ldg(g + i);
}
__device__ __forceinline__ BF4 g_raw(const BF4 *__restrict__ g, idx_t i) {
  const uint2 u = __ldg((const uint2 *)(g + i));
  BF4 b;
  b.x = (unsigned short)(u.x & 0xffffu);
  b.y = (unsigned short)(u.x >> 16);
  b.z = (unsigned short)(u.y & 0xffffu);
  b.w = (unsigned short)(u.y >> 16);
  return b;
}
__device__ __forceinline__ float4 g_value(const float4 &v) { return v; }
__device__ __forceinline__ float4 g_value(const BF4 &b) {
  return make_float4(__uint_as_float((uint32_t)b.x << 16), __uint_as_float((uint32_t)b.y << 16),
                     __uint_as_float((uint32_t)b.z << 16), __uint_as_float((uint32_t)b.w << 16));
}

// ---- compensated accumulation ------------------------------------------------

// Float-float accumulator (Knuth's TwoSum): `hi` carries the running sum,
// `lo` the exact rounding errors of the adds.  Accumulating float products
// this way is about as accurate as the reference's double accumulator
// (optflow4d.cpp:234-241) and costs FP32 adds only; GB300's FP64 rate is a
// small fraction of its FP32 rate.
struct FF {
  float hi, lo;
};
__device__ __forceinline__ void ff_add(FF &a, float p) {
  const float s = a.hi + p;
  const float bp = s - a.hi;
  const float e = (a.hi - (s - bp)) + (p - bp);
  a.hi = s;
  a.lo += e;
}
__device__ __forceinline__ double ff_value(const FF &a) { return (double)a.hi + (double)a.lo; }
// a + b in float-float: TwoSum of the high parts, then a renormalising
// Fast2Sum (Dekker 1971).
__device__ __forceinline__ FF ff_plus(const FF &a, const FF &b) {
  const float s = a.hi + b.hi;
  const float bp = s - a.hi;
  const float e = (a.hi - (s - bp)) + (b.hi - bp);
  const float lo = (a.lo + b.lo) + e;
  const float hi = s + lo;
  return {hi, lo - (hi - s)};
}
__device__ __forceinline__ FF warp_sum_ff(FF v) {
  for (int o = 16; o > 0; o >>= 1) {
    FF b;
    b.hi = __shfl_down_sync(0xffffffffu, v.hi, o);
    b.lo = __shfl_down_sync(0xffffffffu, v.lo, o);
    v = ff_plus(v, b);
  }
  return v;
}

// (float)((double)v * (1./81.)) as the reference computes it
// (knCvExpolBlur4d, optflow4d.cpp:625), mostly without FP64 work.  With
// c = c_hi + c_lo (+ a remainder below 2^-48 c), p + lo approximates v*c to
// about 2^-46 relative and f = RN(p + lo).  Rounding the exact product to
// double and then to float gives f unless the product lies within 2^-53 of
// a float rounding midpoint; products within 2^-40 of a midpoint, and tiny
// or non-finite values, take the double path.
__device__ __forceinline__ float mul_inv81(float v) {
  constexpr double c = 1. / 81.0;
  constexpr float c_hi = (float)c;
  constexpr float c_lo = (float)(c - (double)c_hi);
  const float p = v * c_hi;
  const float pe = __fmaf_rn(v, c_hi, -p);  // v*c_hi - p, exact
  const float lo = __fmaf_rn(v, c_lo, pe);
  const float f = p + lo;
  const unsigned E = (__float_as_uint(f) >> 23) & 0xffu;
  if (E > 41u && E < 255u) {
    const float rem = (p - f) + lo;                       // ~ v*c - f
    const float half_ulp = __uint_as_float((E - 24u) << 23);
    const float margin = __uint_as_float((E - 40u) << 23);
    if (fabsf(fabsf(rem) - half_ulp) > margin) return f;
  } else if (v == 0.f) {
    return f;
  }
  return (float)((double)v * c);
}

// ---- programmatic dependent launch (griddepcontrol, sm_90 and later) -------
// The image gradient g at an interior cell rebuilt from the level's target
// level set i1 with the assembly's own operations (central differences times
// 1/(2 mDx)): the stored g bit for bit, from 4 bytes per cell instead of 16
// (the neighbour loads hit L1 and L2).
struct GradFromI1 {
  const float *__restrict__ i1;
  idx_t sY, sZ, sT;
  float dxf;
  __device__ __forceinline__ float4 operator()(idx_t id) const {
    return make_float4((__ldg(i1 + id + 1) - __ldg(i1 + id - 1)) * dxf,
                       (__ldg(i1 + id + sY) - __ldg(i1 + id - sY)) * dxf,
                       (__ldg(i1 + id + sZ) - __ldg(i1 + id - sZ)) * dxf,
                       (__ldg(i1 + id + sT) - __ldg(i1 + id - sT)) * dxf);
  }
};

// pdl_wait returns once the grid this one depends on has completed and its
// writes are visible (at once for a grid launched without the attribute);
// pdl_launch_dependents lets the next grid of the stream be scheduled, whose
// blocks then wait in their own pdl_wait.  The next grid launches only after
// every block of this one has started or exited, so its waiting blocks never
// hold back this grid's.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Launches a kernel with programmatic stream serialisation, so that its blocks
// are scheduled while the previous kernel of the stream drains (the kernel
// starts with pdl_wait).  Falls back to an ordinary launch if the attribute is
// refused.
template <typename... KArgs, typename... Args>
inline void launch_pdl_smem(void (*k)(KArgs...), dim3 grid, unsigned block, size_t smem,
                            cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, k, args...) != cudaSuccess) {
    cudaGetLastError();
    k<<<grid, block, smem, s>>>(args...);
  }
}
template <typename... KArgs, typename... Args>
inline void launch_pdl(void (*k)(KArgs...), unsigned grid, unsigned block, cudaStream_t s,
                       Args... args) {
  launch_pdl_smem(k, dim3(grid), block, 0, s, args...);
}

// 1 / v for the sums that give beta: the hardware's approximation (off by up to
// a bit, the same way in every cell of equal v) and one Newton step
// r + r (1 - v r), which squares its error and leaves the rounding of the
// result.  Where 1 - v r is no small number (v is 0, infinite or subnormal) the
// approximation stands.  At 64^4 the matvec takes 143.8 us with it, 142.3 with
// the approximation alone and 176 with __frcp_rn.
__device__ __forceinline__ float rcp_newton(float v) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  const float e = __fmaf_rn(-v, r, 1.0f);
  return fabsf(e) < 0.5f ? __fmaf_rn(r, e, r) : r;
}

// a / b in float without the FP64 division (a long chain of dependent FP64
// operations on a part with few FP64 lanes): the float quotient q, off by some
// 2^-22, corrected by its remainder a - q b (Markstein, IBM J. Res. Dev. 34,
// 1990, on divisions with fused multiply-adds).  The remainder is formed in
// FP64 and the correction's own error is some 2^-45 of the result, so this is
// the nearest float of a / b unless a / b lies within 2^-43 of the middle of two.
// Operands or results outside 1e-30 .. 1e30 take the division.
__device__ __forceinline__ float quotient(double a, double b) {
  const float af = (float)a, bf = (float)b;
  const float aa = fabsf(af), ab = fabsf(bf);
  if (aa > 1e-30f && aa < 1e30f && ab > 1e-30f && ab < 1e30f) {
    const float rc = __frcp_rn(bf);
    const float q = af * rc;
    if (fabsf(q) > 1e-30f && fabsf(q) < 1e30f)
      return __fmaf_rn((float)fma(-(double)q, b, a), rc, q);
  }
  return (float)(a / b);
}

// ---- reductions -----------------------------------------------------------

__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_down_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_min(float v) {
  for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_down_sync(0xffffffffu, v, o));
  return v;
}

// Block-wide sum in a fixed tree order; the result is valid in thread 0.
template <int NT>
__device__ __forceinline__ double block_sum(double v, double *sh) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) sh[w] = v;
  __syncthreads();
  if (w == 0) {
    v = (l < NT / 32) ? sh[l] : 0.0;
    v = warp_sum(v);
  }
  __syncthreads();
  return v;
}
// Block sum of float-float values on the FP32 pipe (this part issues FP64
// at about 2 lanes per clock per SM); the result, as a double, is valid in
// thread 0.  sh holds NT / 32 entries.
template <int NT>
__device__ __forceinline__ double block_sum_ff(FF v, FF *sh) {
  v = warp_sum_ff(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) sh[w] = v;
  __syncthreads();
  double r = 0.0;
  if (w == 0) {
    v = (l < NT / 32) ? sh[l] : FF{0.f, 0.f};
    v = warp_sum_ff(v);
    if (l == 0) r = ff_value(v);
  }
  __syncthreads();
  return r;
}
template <int NT>
__device__ __forceinline__ float block_max(float v, float *sh) {
  v = warp_max(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) sh[w] = v;
  __syncthreads();
  if (w == 0) {
    v = (l < NT / 32) ? sh[l] : -INFINITY;
    v = warp_max(v);
  }
  __syncthreads();
  return v;
}
template <int NT>
__device__ __forceinline__ float block_min(float v, float *sh) {
  v = warp_min(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) sh[w] = v;
  __syncthreads();
  if (w == 0) {
    v = (l < NT / 32) ? sh[l] : INFINITY;
    v = warp_min(v);
  }
  __syncthreads();
  return v;
}

// "Last block" completion: every block has published its partial result
// before it increments the counter; the block that sees gridDim.x-1 combines
// the partials in index order (deterministic) and resets the counter.  No
// block ever waits on another.
__device__ __forceinline__ bool last_block_arrives(unsigned int *counter) {
  __shared__ bool is_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned int prev = atomicAdd(counter, 1u);
    is_last = (prev == gridDim.x - 1);
  }
  __syncthreads();
  if (is_last) __threadfence();
  return is_last;
}

}  // namespace flof
