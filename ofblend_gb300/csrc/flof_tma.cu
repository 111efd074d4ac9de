// flof_tma.cu -- TMA-staged slab kernels for the dense 4D stencils on Vec4
// grids: the Gaussian velocity blur (knGaussianBlur, optflow4d.cpp:132-158,
// radius 1 and 2) and the extrapolation sweep (knCvExpolBlur4d, :613-626),
// direct and separable.
//
// Same arithmetic as flof_stencil.cu: every output of the blur and the direct
// sweep sums its (2S+1)^4 neighbourhood in the reference's order (t, z, y, x)
// with float adds in sequence.  A block owns a 32-column (x,y) tile and walks
// the input slabs its output planes need once, in (t, z) order: the blur one
// (z, t) plane per block, the sweeps two z planes walking t with the running
// sums of three t planes in registers.  Each (x,y) slab with its S-cell halo
// is brought into shared memory by one cp.async.bulk.tensor copy issued by a
// single thread, completion signalled on an mbarrier, a few slabs in flight.
// The tensor map views the float4 grid as a 4D float tensor (4X, Y, Z, T), so a
// slab row is one contiguous 16W-byte run, the innermost coordinate 4x is a
// multiple of 16 bytes for every x, and cells outside the grid arrive as
// zeros, which leave a running float sum unchanged (a 16-byte innermost box
// dimension, one float4 per row, made the copies several times slower).
// Lane l of a warp computes column x0+l for RY consecutive rows of
// each plane, so each 8-lane shared-memory phase reads 128 contiguous bytes
// of the dense TMA layout.
//
// Every wait on an mbarrier is bounded; a block that gives up records
// FLOF_DEV_ERR_TMA_TIMEOUT in the context's device error word, waits (again
// bounded) for its copies in flight and returns.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <type_traits>

#include "flof_kernels.h"
#include "flof_tma.cuh"

namespace flof {

namespace {

constexpr int TX = 32;                // tile width: one column per lane

// The sweeps' keep-mask layout: a 16-bit word per thread for RY = 2 rows,
// DZ = 2 z planes and DT = 4 t planes.
struct ExpolGeom {
  static constexpr int RY = 2, DT = 4, DZ = 2;
  static_assert(DZ * DT * RY <= 16, "the keep mask holds 16 cells per thread");
};

// The extrapolation sweeps and the blur add with sm_100-family packed
// `add.rn.f32x2`: a float4 is two float pairs (x,y), (z,w), each lane rounded
// like the scalar add, so the sums are bit for bit the scalar ones in the
// same order at half the instruction count (the FP32 pipe takes the same
// cycles).  The blur's products are packed too, as fma(w, a, -0): the packed
// `mul.rn.f32x2` may be contracted with the add that follows (results differed
// from the separately rounded product in 15% of 4M random cases), while an fma
// whose addend the compiler cannot see cannot; adding -0 leaves the rounded
// product, zeros' signs included.  The -0 is a kernel argument: as a constant
// the fma became a multiply and was contracted after all.
struct __align__(16) P4 {
  unsigned long long lo, hi;
};
__device__ __forceinline__ void add2(unsigned long long &acc, unsigned long long x) {
  asm("add.rn.f32x2 %0, %0, %1;" : "+l"(acc) : "l"(x));
}
__device__ __forceinline__ void acc4(P4 &v, const P4 &a) {
  add2(v.lo, a.lo);
  add2(v.hi, a.hi);
}
__device__ __forceinline__ float4 unpack4(const P4 &v) {
  float4 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v.lo));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.z), "=f"(r.w) : "l"(v.hi));
  return r;
}
__device__ __forceinline__ unsigned long long pair2(float x, float y) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
// the products of two float pairs, each rounded once; nz is the pair (-0, -0)
__device__ __forceinline__ unsigned long long mul2_rn(unsigned long long a, unsigned long long b,
                                                      unsigned long long nz) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(nz));
  return r;
}

template <int S>
__device__ __forceinline__ int clip_code_t(int c, int ext) {
  int lo = S - c;
  lo = lo < 0 ? 0 : lo;
  int hi = c + S - (ext - 1);
  hi = hi < 0 ? 0 : hi;
  return lo * (S + 1) + hi;
}

}  // namespace

struct WTabT {
  float w[40];
};

// The Gaussian blur pass (S = 1, 2).  A block owns an LW-wide (x,y) tile of
// one (z, t) plane and takes the (x,y) slabs of its neighbourhood in the
// reference's (t, z) order; a thread computes RY consecutive rows of one
// column, so every output adds its taps in the reference's sequence.  Slabs
// outside the grid would add products of zero, which leave a running sum
// unchanged, and are not visited.  The tiles cover the output box only.
// Bound by the FP32 pipe: 625 ordered adds per component, plus the products
// w * a, each rounded once as in the reference (mul2_rn) and formed once per
// |yj| for the two rows that use it.  Keeping five output planes' sums, so that
// the products are shared along t too, needs a loop body of 2000 instructions
// and waits for them (no_instruction 2.5 of 4.6 cycles per issue): 2.12 ms at
// 64^4, no faster than this form.
constexpr int BW_NS = 3, BW_MAXW = 4;
template <int LW, int RY>
struct BW {
  static constexpr int RG = 32 / LW;      // row groups of a warp
  static constexpr int UNIT = RG * RY;    // rows of a warp
};
__host__ __device__ constexpr int blur_stride(int w, int h) { return (w * h * 16 + 127) / 128 * 128; }

template <int S, int LW, int RY>
__global__ void __launch_bounds__(32 * BW_MAXW)
k_blur_tma(const __grid_constant__ CUtensorMap map, float4 *__restrict__ dst, Dims4 d, int tiles_x,
           const float *__restrict__ wsum, WTabT wt, unsigned long long nz, int zero_border,
           CellBox box, int *err) {
  using G = BW<LW, RY>;
  constexpr int NS = BW_NS, NV = 2 * S + 1, W = LW + 2 * S;
  extern __shared__ __align__(128) unsigned char raw[];
  __shared__ __align__(8) uint64_t bar[NS];
  __shared__ unsigned long long wsh[40];  // (w, w) pairs
  const int ty_rows = (int)(blockDim.x >> 5) * G::UNIT, h = ty_rows + 2 * S;
  const int stride = blur_stride(W, h);
  const int x0 = box.lo[0] + (int)(blockIdx.x % tiles_x) * LW;
  const int y0 = box.lo[1] + (int)(blockIdx.x / tiles_x) * ty_rows;
  const int z = box.lo[2] + (int)blockIdx.y, t = box.lo[3] + (int)blockIdx.z;
  const int lane = threadIdx.x & 31, lx = lane % LW, x = x0 + lx;
  const int row0 = ((int)(threadIdx.x >> 5) * G::RG + lane / LW) * RY;
  if (threadIdx.x == 0) {
#pragma unroll
    for (int b = 0; b < NS; ++b) mbar_init(&bar[b], 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  for (int i = threadIdx.x; i < 40; i += blockDim.x) wsh[i] = pair2(wt.w[i], wt.w[i]);
  __syncthreads();
  // the slabs inside the grid, t-major
  const int ta = max(t - S, 0), tb = min(t + S, d.t - 1);
  const int za = max(z - S, 0), zb = min(z + S, d.z - 1);
  const int np = (tb - ta + 1) * (zb - za + 1);
  int it = ta, iz = za;  // the next slab to fetch
  auto issue = [&](int p) {
    uint64_t *b = &bar[p % NS];
    mbar_expect_tx(b, (uint32_t)(W * h * 16));
    tma_load_slab(raw + (p % NS) * stride, &map, x0 - S, y0 - S, iz, it, b);
    if (++iz > zb) {
      iz = za;
      ++it;
    }
  };
  if (threadIdx.x == 0)
    for (int p = 0; p < NS - 1 && p < np; ++p) issue(p);

  P4 acc[RY];
#pragma unroll
  for (int q = 0; q < RY; ++q) acc[q] = P4{0ull, 0ull};
  int p = 0;
  for (int tt = ta; tt <= tb; ++tt)
    for (int zz = za; zz <= zb; ++zz, ++p) {
      // buffer (p - 1) % NS was released by the barrier that ended step p - 1
      if (threadIdx.x == 0 && p + NS - 1 < np) issue(p + NS - 1);
      const bool ok = mbar_wait_bounded(&bar[p % NS], (p / NS) & 1);
      // a thread whose wait gave up reads stale values, in bounds; the barrier
      // that ends the step then ends the block
      const P4 *cur = (const P4 *)(raw + (p % NS) * stride) + row0 * W + lx;
      const unsigned long long *wz = wsh + (tt - t) * (tt - t) + (zz - z) * (zz - z);
      // slab row row0 + k feeds output row q via yj = k - q - S
#pragma unroll
      for (int k = 0; k < RY + 2 * S; ++k) {
        P4 a[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i) a[i] = cur[k * W + i];
#pragma unroll
        for (int ay = 0; ay <= S; ++ay) {
          // output rows at y offsets +-ay use the same weights
          const int qm = k - S - ay, qp = k - S + ay;
          if (!((qm >= 0 && qm < RY) || (qp >= 0 && qp < RY))) continue;
          P4 prod[NV];
#pragma unroll
          for (int i = 0; i < NV; ++i) {
            const unsigned long long w2 = wz[ay * ay + (i - S) * (i - S)];
            prod[i] = P4{mul2_rn(w2, a[i].lo, nz), mul2_rn(w2, a[i].hi, nz)};
          }
          if (qm >= 0 && qm < RY)
#pragma unroll
            for (int i = 0; i < NV; ++i) acc4(acc[qm], prod[i]);
          if (ay > 0 && qp >= 0 && qp < RY)
#pragma unroll
            for (int i = 0; i < NV; ++i) acc4(acc[qp], prod[i]);
        }
      }
      if (__syncthreads_or(!ok)) {
        if (threadIdx.x == 0) {
          *(volatile int *)err = FLOF_DEV_ERR_TMA_TIMEOUT;
          // let the copies in flight land before the block's shared memory goes
          for (int r = p; r < np && r < p + NS; ++r) mbar_wait_bounded(&bar[r % NS], (r / NS) & 1);
        }
        __syncthreads();
        return;
      }
    }

  if (x >= box.hi[0]) return;
  constexpr int P1 = (S + 1) * (S + 1);
  const bool zt_inner = z >= 1 && z < d.z - 1 && t >= 1 && t < d.t - 1;
  const int code_zt = (clip_code_t<S>(t, d.t) * P1 + clip_code_t<S>(z, d.z)) * P1;
#pragma unroll
  for (int q = 0; q < RY; ++q) {
    const int y = y0 + row0 + q;
    if (y >= box.hi[1]) continue;
    const idx_t id = d.index(x, y, z, t);
    if (!(zt_inner && x >= 1 && x < d.x - 1 && y >= 1 && y < d.y - 1)) {
      if (zero_border) dst[id] = make_float4(0.f, 0.f, 0.f, 0.f);
      continue;
    }
    const float4 v = unpack4(acc[q]);
    const float ws = __ldg(wsum + (code_zt + clip_code_t<S>(y, d.y)) * P1 + clip_code_t<S>(x, d.x));
    dst[id] = make_float4(v.x / ws, v.y / ws, v.z / ws, v.w / ws);
  }
}

// The extrapolation sweep walking t.  A block owns a 32 x 16 (x,y) tile
// and ETW_DZ consecutive z planes and walks ETW_TC + 2 t planes; for each
// t plane it takes the ETW_DZ + 2 (x,y) slabs (with their one-cell halo)
// that its outputs need, in z order, one TMA copy each, ETW_NS in flight.
// Each thread keeps the running sums of its cells for three output planes
// in registers: slab plane tt adds the taps vt = +1 of output tt - 1 (which
// is then complete and written), vt = 0 of output tt and vt = -1 of output
// tt + 1 (which starts there).  Every output thus adds its 81 taps in the
// reference's order (t, z, y, x) with float adds in sequence, and the loop
// body is the same for every plane: no run-time choice of outputs.
constexpr int ETW_NW = 8, ETW_RY = 2, ETW_DZ = 2, ETW_TC = 8, ETW_NS = 2;
constexpr int ETW_TY = ETW_NW * ETW_RY;
constexpr int ETW_W = TX + 2, ETW_H = ETW_TY + 2;
constexpr int ETW_BYTES = ETW_W * ETW_H * 16;
constexpr int ETW_SPC = 2;  // z slabs per copy of the direct sweep
constexpr int ETW_CBYTES = ETW_SPC * ETW_BYTES;
constexpr int ETW_CSTRIDE = (ETW_CBYTES + 127) / 128 * 128;
constexpr int ETW_SMEM = ETW_NS * ETW_CSTRIDE;
constexpr int ETW_KZ = ETW_DZ + 2;  // slabs per t plane
static_assert(ETW_RY == ExpolGeom::RY && ETW_DZ == ExpolGeom::DZ,
              "the keep mask groups rows and z planes as the sweep does");

// Tiles that a sweep cannot reach.  Before the first sweep every unmarked cell
// holds +0 (knProjectCells leaves it so), and a sweep gives an unmarked cell
// the mean of its 3^4 neighbourhood, so after s sweeps an unmarked cell
// further than s cells (in the maximum norm) from every marked one still holds
// +0: all of its 81 taps were +0, and so is their sum over 81.  dist holds per
// tile a lower bound of that distance; a tile beyond it has nothing to read
// and nothing to write, since both sweep buffers hold +0 there.  The surface
// band is a few cells thick, so the first sweeps of a round touch a part of
// the grid only.
__device__ __forceinline__ bool tile_unreached(const int *__restrict__ dist, int sweep) {
  const size_t tile =
      ((size_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
  return __ldg(dist + tile) > sweep;
}

// Four blocks per SM (64 registers, a few bytes spilled) beat three
// (80 registers): 0.221 against 0.229 ms per 64^4 sweep; copies of two z
// slabs, two copies in flight (one barrier per two slabs), 0.217 ms.
__global__ void __launch_bounds__(32 * ETW_NW, 4)
k_expol_tw(const __grid_constant__ CUtensorMap map, float4 *__restrict__ dst, Dims4 d,
           int tiles_x, const uint16_t *__restrict__ fixed, const int *__restrict__ dist, int sweep,
           int *err) {
  if (tile_unreached(dist, sweep)) return;
  extern __shared__ __align__(128) unsigned char raw[];
  __shared__ __align__(8) uint64_t bar[ETW_NS];
  constexpr int RY = ETW_RY, DZ = ETW_DZ, KZ = ETW_KZ, NS = ETW_NS;
  constexpr int DT = ExpolGeom::DT;  // t planes per keep-mask word
  const int tile = blockIdx.x;
  const int x0 = (tile % tiles_x) * TX, y0 = (tile / tiles_x) * ETW_TY;
  const int z0 = blockIdx.y * DZ, t0 = blockIdx.z * ETW_TC;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int x = x0 + tx;
  const int ygroups = (d.y + RY - 1) / RY, zgroups = (d.z + DZ - 1) / DZ;
  const int yg = y0 / RY + ty;
  const bool xy_ok = x < d.x && yg < ygroups;
  if (threadIdx.x == 0) {
#pragma unroll
    for (int b = 0; b < NS; ++b) mbar_init(&bar[b], 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  constexpr int CPP = KZ / ETW_SPC;   // copies per t plane
  // copy p: plane t0 - 1 + p / CPP, slabs from z0 - 1 + SPC (p % CPP)
  const int NP = (ETW_TC + 2) * CPP;
  auto issue = [&](int p) {
    uint64_t *b = &bar[p % NS];
    mbar_expect_tx(b, ETW_CBYTES);
    tma_load_slab(raw + (p % NS) * ETW_CSTRIDE, &map, x0 - 1, y0 - 1, z0 - 1 + ETW_SPC * (p % CPP),
                  t0 - 1 + p / CPP, b);
  };
  if (threadIdx.x == 0) {
#pragma unroll
    for (int p = 0; p < NS - 1; ++p) issue(p);
  }
  // running sums of outputs tt - 1 (A), tt (B) and tt + 1 (C)
  P4 A[DZ][RY], B[DZ][RY], C[DZ][RY];
  // One t plane j (tt = t0 - 1 + j).  SA, SB, SC say which of the three
  // outputs lie in the block's range t0 .. t0 + ETW_TC - 1: the first two and
  // the last two planes skip the sums of the others (a fifth of the adds).
  auto plane = [&](int j, auto SA, auto SB, auto SC) -> bool {
    constexpr bool DA = decltype(SA)::value, DB = decltype(SB)::value, DC = decltype(SC)::value;
    if (DC) {
#pragma unroll
      for (int oz = 0; oz < DZ; ++oz)
#pragma unroll
        for (int q = 0; q < RY; ++q) memset(&C[oz][q], 0, sizeof(P4));
    }
#pragma unroll
    for (int zc = 0; zc < CPP; ++zc) {
      const int p = j * CPP + zc;
      // buffer (p - 1) % NS was released by the barrier that ended copy p - 1
      if (threadIdx.x == 0 && p + NS - 1 < NP) issue(p + NS - 1);
      // A thread whose wait gave up still reads the buffer (stale values, in
      // bounds); the barrier that ends the copy's step then ends the block.
      const bool ok = mbar_wait_bounded(&bar[p % NS], (p / NS) & 1);
#pragma unroll
      for (int sl = 0; sl < ETW_SPC; ++sl) {
        const int zk = zc * ETW_SPC + sl;
        const P4 *cur = (const P4 *)(raw + (p % NS) * ETW_CSTRIDE + sl * ETW_BYTES);
#pragma unroll
        for (int k = 0; k < RY + 2; ++k) {
          const P4 *row = cur + (RY * ty + k) * ETW_W + tx;
          const P4 a0 = row[0], a1 = row[1], a2 = row[2];
#pragma unroll
          for (int oz = 0; oz < DZ; ++oz) {
            const int zrel = zk - 1 - oz;  // this slab's z offset from output plane z0 + oz
            if (zrel < -1 || zrel > 1) continue;
#pragma unroll
            for (int q = 0; q < RY; ++q) {
              const int yj = k - q - 1;
              if (yj < -1 || yj > 1) continue;
              // vt = -1 of output tt + 1, vt = 0 of output tt, vt = +1 of output tt - 1
              if (DC) {
                acc4(C[oz][q], a0);
                acc4(C[oz][q], a1);
                acc4(C[oz][q], a2);
              }
              if (DB) {
                acc4(B[oz][q], a0);
                acc4(B[oz][q], a1);
                acc4(B[oz][q], a2);
              }
              if (DA) {
                acc4(A[oz][q], a0);
                acc4(A[oz][q], a1);
                acc4(A[oz][q], a2);
              }
            }
          }
        }
      }
      if (__syncthreads_or(!ok)) {
        if (threadIdx.x == 0) {
          *(volatile int *)err = FLOF_DEV_ERR_TMA_TIMEOUT;
          for (int r = p; r < NP && r < p + NS; ++r) mbar_wait_bounded(&bar[r % NS], (r / NS) & 1);
        }
        __syncthreads();
        return false;
      }
    }
    // output tt - 1 = t0 - 2 + j is complete
    const int t = t0 - 2 + j;
    if (DA && xy_ok && t < d.t) {
      const unsigned keep =
          __ldg(fixed + (((size_t)(t / DT) * zgroups + blockIdx.y) * ygroups + yg) * d.x + x);
#pragma unroll
      for (int oz = 0; oz < DZ; ++oz) {
        const int z = z0 + oz;
        if (z >= d.z) break;
#pragma unroll
        for (int q = 0; q < RY; ++q) {
          const int y = y0 + RY * ty + q;
          if (y >= d.y) continue;
          if (keep >> ((oz * DT + t % DT) * RY + q) & 1u) continue;
          const float4 v = unpack4(A[oz][q]);
          dst[d.index(x, y, z, t)] =
              make_float4(mul_inv81(v.x), mul_inv81(v.y), mul_inv81(v.z), mul_inv81(v.w));
        }
      }
    }
#pragma unroll
    for (int oz = 0; oz < DZ; ++oz)
#pragma unroll
      for (int q = 0; q < RY; ++q) {
        A[oz][q] = B[oz][q];
        B[oz][q] = C[oz][q];
      }
    return true;
  };
  using T_ = std::true_type;
  using F_ = std::false_type;
  static_assert(ETW_TC >= 2, "the peeled planes are distinct");
  if (!plane(0, F_(), F_(), T_())) return;
  if (!plane(1, F_(), T_(), T_())) return;
  for (int j = 2; j < ETW_TC; ++j)
    if (!plane(j, T_(), T_(), T_())) return;
  if (!plane(ETW_TC, T_(), T_(), F_())) return;
  plane(ETW_TC + 1, T_(), F_(), F_());
}

// Per brick of BRICK_X x 8 x 8 x 8 cells, the bounds of its marked cells in
// x, y, z, t (lo > hi: none).
constexpr int BRICK_X = 16, BRICK = 8;
struct BrickBounds {
  int lo[4], hi[4];
};
__global__ void __launch_bounds__(128)
k_expol_bricks(const float *__restrict__ mark, BrickBounds *__restrict__ out, Dims4 d, int bx,
               int by, int bz) {
  __shared__ int sh[8];
  if (threadIdx.x < 8) sh[threadIdx.x] = threadIdx.x < 4 ? 0x7fffffff : -1;
  __syncthreads();
  const int xb = blockIdx.x % bx, r = blockIdx.x / bx, yb = r % by, r2 = r / by;
  const int zb = r2 % bz, tb = r2 / bz;
  const int x = xb * BRICK_X + (threadIdx.x & 15), y = yb * BRICK + (threadIdx.x >> 4);
  int lo[4] = {0x7fffffff, 0x7fffffff, 0x7fffffff, 0x7fffffff}, hi[4] = {-1, -1, -1, -1};
  if (x < d.x && y < d.y)
    for (int t = tb * BRICK; t < min(tb * BRICK + BRICK, d.t); ++t)
      for (int z = zb * BRICK; z < min(zb * BRICK + BRICK, d.z); ++z)
        if (__ldg(mark + d.index(x, y, z, t)) != 0.f) {
          const int c[4] = {x, y, z, t};
#pragma unroll
          for (int a = 0; a < 4; ++a) {
            lo[a] = min(lo[a], c[a]);
            hi[a] = max(hi[a], c[a]);
          }
        }
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    lo[a] = __reduce_min_sync(0xffffffffu, lo[a]);
    hi[a] = __reduce_max_sync(0xffffffffu, hi[a]);
    if ((threadIdx.x & 31) == 0) {
      atomicMin(&sh[a], lo[a]);
      atomicMax(&sh[4 + a], hi[a]);
    }
  }
  __syncthreads();
  if (threadIdx.x < 8) ((int *)(out + blockIdx.x))[threadIdx.x] = sh[threadIdx.x];
}

// dist[tile]: the least distance in the maximum norm between the tile's
// outputs and a brick's bounds (marked cells lie within those).
__global__ void __launch_bounds__(128)
k_expol_dist(const BrickBounds *__restrict__ b, int nb, int *__restrict__ dist, int tiles_x) {
  __shared__ int best;
  if (threadIdx.x == 0) best = 0x7fffffff;
  __syncthreads();
  const int lo[4] = {(int)(blockIdx.x % tiles_x) * TX, (int)(blockIdx.x / tiles_x) * ETW_TY,
                     (int)blockIdx.y * ETW_DZ, (int)blockIdx.z * ETW_TC};
  const int hi[4] = {lo[0] + TX - 1, lo[1] + ETW_TY - 1, lo[2] + ETW_DZ - 1, lo[3] + ETW_TC - 1};
  int mine = 0x7fffffff;
  for (int k = threadIdx.x; k < nb; k += 128) {
    const int4 l = __ldg((const int4 *)(b + k)), h = __ldg((const int4 *)(b + k) + 1);
    if (h.x < 0) continue;
    int g = max(l.x - hi[0], lo[0] - h.x);
    g = max(g, max(l.y - hi[1], lo[1] - h.y));
    g = max(g, max(l.z - hi[2], lo[2] - h.z));
    g = max(g, max(l.w - hi[3], lo[3] - h.w));
    mine = min(mine, g);
  }
  mine = __reduce_min_sync(0xffffffffu, mine);
  if ((threadIdx.x & 31) == 0) atomicMin(&best, mine);
  __syncthreads();
  if (threadIdx.x == 0)
    dist[((size_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = best;
}

// The separable extrapolation sweep (blurType 2) walking t.  It takes
// k_expol_tw's slabs in k_expol_tw's order but forms each output's 3^4 sum as
// box sums: per slab the x sums of the rows a thread needs and the y sums of
// three of those, added over the three z slabs of each output plane as the
// slabs arrive, and over three consecutive t planes from a register ring.
// Each sum is taken in the two-pass separable sweep's order (x, then y, z, t,
// each (a-1 + a0) + a+1), so the two give the same bits; a cell costs about
// sixteen float4 adds instead of 81.  The kernel is bound by latency (few
// warps, two dependent shared-memory and add steps per slab) more than by
// shared-memory or DRAM bandwidth, so warps count most: at 64^4 on GB300,
// RY = 2 rows per thread (8 warps, three blocks per SM) took 0.168 ms a
// sweep against 0.178 ms for RY = 4 (4 warps), and TC = 4 or deeper slab
// pipelines did not help.  A copy brings two z slabs (one block barrier per
// two slabs): 0.165 ms.
constexpr int ESW_RY = 2, ESW_NW = ETW_TY / ESW_RY, ESW_TC = 8, ESW_NS = 3, ESW_MINB = 3;
static_assert(ESW_TC == ETW_TC, "both sweeps have the tiles that k_expol_dist measures");
constexpr int ESW_SPC = 2;  // z slabs per copy: one barrier step per two slabs
constexpr int ESW_CBYTES = ESW_SPC * ETW_BYTES;  // one copy, its slabs back to back
constexpr int ESW_CSTRIDE = (ESW_CBYTES + 127) / 128 * 128;
constexpr int ESW_SMEM = ESW_NS * ESW_CSTRIDE;
static_assert(ETW_KZ % ESW_SPC == 0, "whole copies per plane");

__global__ void __launch_bounds__(32 * ESW_NW, ESW_MINB)
k_expol_sep_tw(const __grid_constant__ CUtensorMap map, float4 *__restrict__ dst, Dims4 d,
               int tiles_x, const uint16_t *__restrict__ fixed, const int *__restrict__ dist,
               int sweep, int *err) {
  if (tile_unreached(dist, sweep)) return;
  extern __shared__ __align__(128) unsigned char raw[];
  __shared__ __align__(8) uint64_t bar[ESW_NS];
  constexpr int RY = ESW_RY, DZ = ETW_DZ, KZ = ETW_KZ, NS = ESW_NS;
  constexpr int MRY = ExpolGeom::RY, DT = ExpolGeom::DT;  // keep-mask word geometry
  static_assert(RY % MRY == 0, "a thread's rows cover whole keep-mask row groups");
  static_assert((DT & (DT - 1)) == 0, "t % DT as a mask");
  const int tile = blockIdx.x;
  const int x0 = (tile % tiles_x) * TX, y0 = (tile / tiles_x) * ETW_TY;
  const int z0 = blockIdx.y * DZ, t0 = blockIdx.z * ESW_TC;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int x = x0 + tx;
  const int ygroups = (d.y + MRY - 1) / MRY, zgroups = (d.z + DZ - 1) / DZ;
  if (threadIdx.x == 0) {
#pragma unroll
    for (int b = 0; b < NS; ++b) mbar_init(&bar[b], 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  constexpr int CPP = KZ / ESW_SPC;   // copies per t plane
  // copy p: plane t0 - 1 + p / CPP, slabs from z0 - 1 + SPC (p % CPP)
  const int NP = (ESW_TC + 2) * CPP;
  auto issue = [&](int p) {
    uint64_t *b = &bar[p % NS];
    mbar_expect_tx(b, ESW_CBYTES);
    tma_load_slab(raw + (p % NS) * ESW_CSTRIDE, &map, x0 - 1, y0 - 1, z0 - 1 + ESW_SPC * (p % CPP),
                  t0 - 1 + p / CPP, b);
  };
  if (threadIdx.x == 0) {
#pragma unroll
    for (int p = 0; p < NS - 1; ++p) issue(p);
  }
  // z sums of planes tt - 2 (Z0), tt - 1 (Z1) and tt (Zc, filled slab by slab)
  P4 Z0[DZ][RY], Z1[DZ][RY], Zc[DZ][RY];
  for (int j = 0; j < ESW_TC + 2; ++j) {
    // keep-mask words of output plane t = t0 - 2 + j, loaded before its slabs
    // are summed (all ones: nothing to write)
    const int t = t0 - 2 + j;
    unsigned keep[RY / MRY];
#pragma unroll
    for (int g = 0; g < RY / MRY; ++g) {
      const int yb = y0 + RY * ty + g * MRY;
      keep[g] = 0xffffu;
      if (j >= 2 && x < d.x && t < d.t && yb < d.y)
        keep[g] = __ldg(fixed + ((((size_t)(t / DT) * zgroups + blockIdx.y) * ygroups + yb / MRY) *
                                     d.x + x));
    }
#pragma unroll
    for (int zc = 0; zc < CPP; ++zc) {
      const int p = j * CPP + zc;
      if (threadIdx.x == 0 && p + NS - 1 < NP) issue(p + NS - 1);
      // A thread whose wait gave up still reads the buffer (stale values,
      // in bounds); the barrier that ends the copy's step then ends the block.
      const bool ok = mbar_wait_bounded(&bar[p % NS], (p / NS) & 1);
#pragma unroll
      for (int sl = 0; sl < ESW_SPC; ++sl) {
        const int zk = zc * ESW_SPC + sl;
        const P4 *cur =
            (const P4 *)(raw + (p % NS) * ESW_CSTRIDE + sl * ETW_BYTES) + RY * ty * ETW_W + tx;
        auto xsum = [&](int k) {
          const P4 *row = cur + k * ETW_W;
          P4 v = row[0];
          acc4(v, row[1]);
          acc4(v, row[2]);
          return v;
        };
        P4 r0 = xsum(0), r1 = xsum(1);
#pragma unroll
        for (int q = 0; q < RY; ++q) {
          const P4 r2 = xsum(q + 2);
          P4 xy = r0;
          acc4(xy, r1);
          acc4(xy, r2);
#pragma unroll
          for (int oz = 0; oz < DZ; ++oz) {
            const int zrel = zk - 1 - oz;  // this slab's z offset from output plane z0 + oz
            if (zrel == -1) Zc[oz][q] = xy;
            else if (zrel <= 1) acc4(Zc[oz][q], xy);
          }
          r0 = r1;
          r1 = r2;
        }
      }
      if (__syncthreads_or(!ok)) {
        if (threadIdx.x == 0) {
          *(volatile int *)err = FLOF_DEV_ERR_TMA_TIMEOUT;
          for (int r = p; r < NP && r < p + NS; ++r) mbar_wait_bounded(&bar[r % NS], (r / NS) & 1);
        }
        __syncthreads();
        return;
      }
    }
    // output plane t: (Z(t - 1) + Z(t)) + Z(t + 1).  A clear bit means an
    // unmarked interior cell, so x, y, z and t are then inside the grid.
#pragma unroll
    for (int g = 0; g < RY / MRY; ++g) {
      const int yb = y0 + RY * ty + g * MRY;
#pragma unroll
      for (int oz = 0; oz < DZ; ++oz) {
#pragma unroll
        for (int m = 0; m < MRY; ++m) {
          if (keep[g] >> ((oz * DT + (t & (DT - 1))) * MRY + m) & 1u) continue;
          const int q = g * MRY + m;
          P4 v = Z0[oz][q];
          acc4(v, Z1[oz][q]);
          acc4(v, Zc[oz][q]);
          const float4 s = unpack4(v);
          dst[d.index(x, yb + m, z0 + oz, t)] =
              make_float4(mul_inv81(s.x), mul_inv81(s.y), mul_inv81(s.z), mul_inv81(s.w));
        }
      }
    }
#pragma unroll
    for (int oz = 0; oz < DZ; ++oz)
#pragma unroll
      for (int q = 0; q < RY; ++q) {
        Z0[oz][q] = Z1[oz][q];
        Z1[oz][q] = Zc[oz][q];
      }
  }
}

namespace {

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  // looked up once (thread-safe static init); null when the driver lacks it
  static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                         &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      return (PFN_cuTensorMapEncodeTiled_v12000)p;
    cudaGetLastError();
    return (PFN_cuTensorMapEncodeTiled_v12000) nullptr;
  }();
  return fn;
}

}  // namespace

// Tensor map of a float4 grid as a 4D float tensor (4X, Y, Z, T) with a
// (4W, H, 1, 1) box: each slab row is one contiguous run of 16W bytes.
bool encode_slab_map(CUtensorMap *m, const float4 *base, Dims4 d, int W, int H, int D) {
  PFN_cuTensorMapEncodeTiled_v12000 fn = encode_fn();
  if (!fn || ((uintptr_t)base & 15) || 4 * W > 256) return false;
  const cuuint64_t dims[4] = {(cuuint64_t)4 * d.x, (cuuint64_t)d.y, (cuuint64_t)d.z,
                              (cuuint64_t)d.t};
  const cuuint64_t strides[3] = {(cuuint64_t)16 * d.x, (cuuint64_t)16 * d.x * d.y,
                                 (cuuint64_t)16 * d.x * d.y * d.z};
  const cuuint32_t box[4] = {(cuuint32_t)(4 * W), (cuuint32_t)H, (cuuint32_t)D, 1};
  const cuuint32_t es[4] = {1, 1, 1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (void *)base, dims, strides, box, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

namespace {

// The shape of a blur launch: tile width, rows per thread, warps per block.
struct BlurShape {
  int lw, ry, nw, ny;
};
// Of 32, 16 and 8 columns and 8 or 4 rows a thread, the tile that computes the
// least: cells beyond the box are computed like the others (tiles of 32 x 32
// computed 1.8 times the cells at 48^4, 2.6 times at 40^3), and the products
// shared between rows make a row of 8 cheaper than one of 4 (175 against 190
// pipe cycles a slab).  A grid with fewer than three warps per SM partition at
// 8 rows takes 4, for more warps.
BlurShape blur_shape(const CellBox &box) {
  const Dims4 d{box.hi[0] - box.lo[0], box.hi[1] - box.lo[1], box.hi[2] - box.lo[2],
                box.hi[3] - box.lo[3]};
  BlurShape best = {32, 8, 4, 1};
  double bt = 0.0;
  for (int ry : {8, 4})
    for (int lw : {32, 16, 8}) {
      const int unit = 32 / lw * ry;
      const int ny = (d.y + BW_MAXW * unit - 1) / (BW_MAXW * unit);
      const int nw = ((d.y + ny - 1) / ny + unit - 1) / unit;
      const double warps = (double)((d.x + lw - 1) / lw) * ny * nw * d.z * d.t;
      const double slots = 4.0 * sm_count(), row = ry == 8 ? 175.0 : 190.0;
      // with few warps per partition their latency shows
      const double per = warps / slots, t = row * ry * (per < 3.0 ? 1.0 + per * 2.0 / 3.0 : per);
      if (bt == 0.0 || t < bt) {
        bt = t;
        best = BlurShape{lw, ry, nw, ny};
      }
    }
  return best;
}

template <int S, int LW, int RY>
bool launch_blur_shape(const float4 *src, float4 *dst, Dims4 d, const float *wsum, const WTabT &wt,
                       int zero_border, const CellBox &box, int *err, cudaStream_t st,
                       const BlurShape &b) {
  constexpr int W = LW + 2 * S, UNIT = BW<LW, RY>::UNIT;
  const int tiles_x = (box.hi[0] - box.lo[0] + LW - 1) / LW, h = b.nw * UNIT + 2 * S;
  CUtensorMap map;
  if (!encode_slab_map(&map, src, d, W, h)) return false;
  if (allow_smem<k_blur_tma<S, LW, RY>>(BW_NS * blur_stride(W, BW_MAXW * UNIT + 2 * S)) !=
      cudaSuccess)
    return false;
  const dim3 grid(tiles_x * b.ny, box.hi[2] - box.lo[2], box.hi[3] - box.lo[3]);
  k_blur_tma<S, LW, RY><<<grid, 32 * b.nw, BW_NS * blur_stride(W, h), st>>>(
      map, dst, d, tiles_x, wsum, wt, 0x8000000080000000ull, zero_border, box, err);
  return true;
}

template <int S>
bool launch_blur(const float4 *src, float4 *dst, Dims4 d, const float *wsum, const float *w,
                 int zero_border, const CellBox &box, int *err, cudaStream_t st) {
  if (d.z > 65535 || d.t > 65535) return false;
  if (box.cells() == 0) return true;
  WTabT wt;
  for (int i = 0; i < 40; ++i) wt.w[i] = (w && i <= 4 * S * S) ? w[i] : 0.f;
  const BlurShape b = blur_shape(box);
#define FLOF_BLUR(LW, RY) \
  if (b.lw == LW && b.ry == RY) return launch_blur_shape<S, LW, RY>(src, dst, d, wsum, wt, zero_border, box, err, st, b)
  FLOF_BLUR(32, 8);
  FLOF_BLUR(16, 8);
  FLOF_BLUR(8, 8);
  FLOF_BLUR(32, 4);
  FLOF_BLUR(16, 4);
  FLOF_BLUR(8, 4);
#undef FLOF_BLUR
  return false;
}

}  // namespace

bool launch_gauss_tma(const float4 *src, float4 *dst, Dims4 d, int s, const float *wtab,
                      const float *wsum_dev, int zero_border, const CellBox &box, int *err,
                      cudaStream_t st) {
  if (s == 1) return launch_blur<1>(src, dst, d, wsum_dev, wtab, zero_border, box, err, st);
  if (s == 2) return launch_blur<2>(src, dst, d, wsum_dev, wtab, zero_border, box, err, st);
  return false;
}

namespace {

// One 16-bit word per sweep thread: (x, y group of RY rows, z group of DZ, t
// group of DT), x fastest.  A bit is set for each of the thread's cells that
// the sweep leaves alone: marked, outside the interior (knCvExpolBlur4d runs
// over bnd = 1), or past the grid's end.
__global__ void k_expol_mask(const float *__restrict__ mark, uint16_t *__restrict__ mask, Dims4 d,
                             int ygroups, int zgroups, long long nwords) {
  constexpr int RY = ExpolGeom::RY, DT = ExpolGeom::DT, DZ = ExpolGeom::DZ;
  for (long long w = blockIdx.x * (long long)blockDim.x + threadIdx.x; w < nwords;
       w += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(w % d.x);
    long long r = w / d.x;
    const int yg = (int)(r % ygroups);
    r /= ygroups;
    const int zg = (int)(r % zgroups);
    const int tg = (int)(r / zgroups);
    unsigned bits = 0;
    for (int oz = 0; oz < DZ; ++oz)
      for (int o = 0; o < DT; ++o)
        for (int q = 0; q < RY; ++q) {
          const int y = yg * RY + q, z = zg * DZ + oz, t = tg * DT + o;
          if (y >= d.y || z >= d.z || t >= d.t) {
            bits |= 1u << ((oz * DT + o) * RY + q);
            continue;
          }
          const bool inner = x >= 1 && x < d.x - 1 && y >= 1 && y < d.y - 1 && z >= 1 &&
                             z < d.z - 1 && t >= 1 && t < d.t - 1;
          if (!inner || __ldg(mark + d.index(x, y, z, t)) != 0.f)
            bits |= 1u << ((oz * DT + o) * RY + q);
        }
    mask[w] = (uint16_t)bits;
  }
}

}  // namespace

size_t expol_mask_words(Dims4 d) {
  return (size_t)d.x * ((d.y + ExpolGeom::RY - 1) / ExpolGeom::RY) *
         ((d.z + ExpolGeom::DZ - 1) / ExpolGeom::DZ) * ((d.t + ExpolGeom::DT - 1) / ExpolGeom::DT);
}

void launch_expol_mask(const float *mark, uint16_t *mask, Dims4 d, cudaStream_t st) {
  const long long n = (long long)expol_mask_words(d);
  const int ygroups = (d.y + ExpolGeom::RY - 1) / ExpolGeom::RY;
  const int zgroups = (d.z + ExpolGeom::DZ - 1) / ExpolGeom::DZ;
  k_expol_mask<<<grid_for(n, 256), 256, 0, st>>>(mark, mask, d, ygroups, zgroups, n);
}

namespace {
dim3 sweep_grid(Dims4 d) {
  const int tiles_x = (d.x + TX - 1) / TX, tiles_y = (d.y + ETW_TY - 1) / ETW_TY;
  return dim3(tiles_x * tiles_y, (d.z + ETW_DZ - 1) / ETW_DZ, (d.t + ETW_TC - 1) / ETW_TC);
}
int brick_count(Dims4 d, int *bx, int *by, int *bz) {
  *bx = (d.x + BRICK_X - 1) / BRICK_X;
  *by = (d.y + BRICK - 1) / BRICK;
  *bz = (d.z + BRICK - 1) / BRICK;
  return *bx * *by * *bz * ((d.t + BRICK - 1) / BRICK);
}
}  // namespace

size_t expol_reach_bytes(Dims4 d) {
  int bx, by, bz;
  const dim3 g = sweep_grid(d);
  return sizeof(BrickBounds) * (size_t)brick_count(d, &bx, &by, &bz) +
         sizeof(int) * (size_t)g.x * g.y * g.z;
}

const int *launch_expol_reach(const float *mark, void *scratch, Dims4 d, cudaStream_t st) {
  int bx, by, bz;
  const int nb = brick_count(d, &bx, &by, &bz);
  const dim3 g = sweep_grid(d);
  BrickBounds *b = (BrickBounds *)scratch;
  int *dist = (int *)(b + nb);
  if (g.y > 65535 || g.z > 65535) return dist;  // the sweeps refuse such a grid too
  k_expol_bricks<<<nb, 128, 0, st>>>(mark, b, d, bx, by, bz);
  k_expol_dist<<<g, 128, 0, st>>>(b, nb, dist, (d.x + TX - 1) / TX);
  return dist;
}

bool launch_expol_tw(const float4 *in, float4 *out, const uint16_t *mask, const int *dist,
                     int sweep, Dims4 d, int *err, cudaStream_t st) {
  const dim3 grid = sweep_grid(d);
  if (grid.y > 65535 || grid.z > 65535) return false;
  CUtensorMap map;
  if (!encode_slab_map(&map, in, d, ETW_W, ETW_H, ETW_SPC)) return false;
  if (allow_smem<k_expol_tw>(ETW_SMEM) != cudaSuccess) return false;
  k_expol_tw<<<grid, 32 * ETW_NW, ETW_SMEM, st>>>(map, out, d, (d.x + TX - 1) / TX, mask, dist,
                                                  sweep, err);
  return true;
}

bool launch_expol_sep_tw(const float4 *in, float4 *out, const uint16_t *mask, const int *dist,
                         int sweep, Dims4 d, int *err, cudaStream_t st) {
  const dim3 grid = sweep_grid(d);
  if (grid.y > 65535 || grid.z > 65535) return false;
  CUtensorMap map;
  if (!encode_slab_map(&map, in, d, ETW_W, ETW_H, ESW_SPC)) return false;
  if (allow_smem<k_expol_sep_tw>(ESW_SMEM) != cudaSuccess) return false;
  k_expol_sep_tw<<<grid, 32 * ESW_NW, ESW_SMEM, st>>>(map, out, d, (d.x + TX - 1) / TX, mask,
                                                      dist, sweep, err);
  return true;
}

}  // namespace flof
