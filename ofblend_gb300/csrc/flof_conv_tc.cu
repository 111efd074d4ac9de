// flof_conv_tc.cu -- the learned warm start's 3^4 convolutions on the
// tcgen05 tensor cores: forward, input gradient and weight gradient as
// implicit GEMMs of 128-row tiles, accumulated in tensor memory.
//
// Operands: the weights are BF16 already (rounded from the FP32 master
// weights), so they enter as they are.  Activations and gradients are FP32;
// each value x enters as two BF16 parts hi = bf16(x), lo = bf16(x - hi)
// (about 16 significant bits), so the products carry FP32-like accuracy:
//   forward / input gradient: acc += A_hi W + A_lo W            (2 MMAs)
//   weight gradient:          acc += A_hi B_hi + A_lo B_hi + A_hi B_lo (3 MMAs)
// with FP32 accumulation in tensor memory.
//
// Stride-1 gradients read each operand value once per tile (k_dgrad_halo,
// k_wgrad_halo below).  The forward pass and the stride-2 gradients (k_conv_tc)
// are implicit GEMMs over an im2col gather.
//
// k_conv_tc, per block: 256 threads gather a 128 x 64 reduction chunk of the operand
// (im2col on the fly: voxel rows x (tap, channel), or (tap, channel) rows x
// voxels for the weight gradient) through registers into shared memory in
// the 128-byte-swizzled K-major layout (flof_tcgen05.cuh), while the
// previous chunk's MMAs (issued by a ninth warp) run; two stages, each released by a
// tcgen05.commit on its mbarrier.  The forward and input-gradient gathers
// run along channels (16 lanes read 256 contiguous bytes of a row), the
// weight-gradient gather along the (tap, channel) rows.  The weight
// gradient carries one more row of ones, whose products are the bias
// gradient.  Layers with few row tiles split the reduction into slices
// written to a work buffer and summed in slice order (deterministic), with
// the bias and ReLU applied there.
//
// Every mbarrier wait is bounded: a block that gives up stores
// FLOF_DEV_ERR_TC_TIMEOUT in the context's device error word, waits (again
// bounded) for its issued MMAs, frees its tensor memory and returns.
#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>

#include "flof_internal.h"
#include "flof_tcgen05.cuh"

namespace flof {

namespace {

using namespace tc;

constexpr int TB_M = 128;  // rows per block (the MMA's M)
constexpr int TB_K = 64;   // reduction entries per chunk (four K = 16 MMAs)
constexpr int TB_T = 256;  // threads that stage operands
constexpr int TB_W = TB_T + 32;  // plus one warp that issues the MMAs
constexpr int KG_T = 8 * TB_M / TB_T;  // weight gradient: reduction groups (of 8) per thread
constexpr int A_TILE = TB_M * TB_K * 2;  // bytes of one BF16 A tile

struct TcArgs {
  const float *A;         // MODE 0: input; MODE 1: output gradient; MODE 2: input
  const float *B32;       // MODE 2: output gradient
  const uint16_t *Bw;     // MODE 0: WT[cout][Kpad]; MODE 1: WB[tap][cin][cout] (BF16 bits)
  const float *bias;      // MODE 0, unsplit only
  float *C;               // result rows x N, or slices of it
  int *err;
  int rin, rout, cin, cout, stride;
  int M, N, K, Kpad;      // rows, columns, reduction length, WT row length
  int relu, kslice, ncols;
  int bias_row;           // MODE 2: the last row is all ones (the bias gradient)
  NetGradEpi epi;         // MODE 1, unsplit only
};

// A tap of the reduction: its source voxel is the row's voxel plus `off`
// (linear, in the grid the tap reads), and it falls off that grid for rows
// whose edge mask shares a bit with `need`.  For a forward tap with offsets
// o in 0..2 per axis, `need` has bit a where o_a = 0 and bit 4 + a where
// o_a = 2, and off = sum (o_a - 1) stride_a.  Bit 8 is always set, so an
// invalid row (edge mask 0x100) reads nothing.
struct TapEnt {
  int need, off;
};

__device__ const float kOne = 1.f;  // the weight gradient's bias row

__device__ __forceinline__ void tap_digits(int tap, int o[4]) {
  o[0] = tap % 3;
  o[1] = (tap / 3) % 3;
  o[2] = (tap / 9) % 3;
  o[3] = tap / 27;
}

// edge mask of a source position s (per axis, s = coordinate * stride): bit
// a when s_a = 0 (offset 0 falls off), bit 4 + a when s_a + 1 >= ext
__device__ __forceinline__ int edge_mask(const int s[4], int ext) {
  int m = 0;
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    m |= (s[a] == 0) << a;
    m |= (s[a] + 1 >= ext) << (4 + a);
  }
  return m;
}

// weight gradient: voxel table of reduction chunk c (its 64 output voxels):
// (input voxel of v * stride times cin, edge mask), bit 8 set past the
// slice's end
__device__ __forceinline__ void fill_vtab(int2 *vt, int tid, int kbeg, int c, int nch, int kend,
                                          int rout, int rin, int stride, int cin) {
  if (tid >= TB_K) return;
  const int v = kbeg + c * TB_K + tid;
  int2 e = make_int2(0, 0x100);
  if (c < nch && v < kend) {
    int s[4], q = v;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      s[a] = (q % rout) * stride;
      q /= rout;
    }
    e = make_int2((s[0] + rin * (s[1] + rin * (s[2] + rin * s[3]))) * cin, edge_mask(s, rin));
  }
  vt[tid] = e;
}

// MODE 0/1 gather: this thread's four channels, starting at reduction index
// k (of K), of rows rsub, rsub + 16, ... of the tile: zero where the tap's
// `need` mask meets the row's edge mask or k is past the end
template <int VEC>
__device__ __forceinline__ void gather01(float4 (&xv)[TB_M / 16], const float *__restrict__ A,
                                         int k, int K, const TapEnt *taps, const int2 *rows_s,
                                         int rsub, int ch) {
#pragma unroll
  for (int it = 0; it < TB_M / 16; ++it) xv[it] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (VEC) {
    if (k >= K) return;
    const int tap = k / ch, c = k - tap * ch;
    const TapEnt t = taps[tap];
#pragma unroll
    for (int it = 0; it < TB_M / 16; ++it) {
      const int2 ri = rows_s[it * 16 + rsub];
      if (!(ri.y & t.need))
        xv[it] = __ldg(reinterpret_cast<const float4 *>(A + (size_t)(ri.x + t.off) * ch + c));
    }
  } else {  // a channel count that is not a multiple of 8 (the forward pass only)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int kj = k + j;
      if (kj < K) {
        const int tap = kj / ch, ci = kj - tap * ch;
        const TapEnt t = taps[tap];
#pragma unroll
        for (int it = 0; it < TB_M / 16; ++it) {
          const int2 ri = rows_s[it * 16 + rsub];
          if (!(ri.y & t.need)) {
            const float v = __ldg(A + (size_t)(ri.x + t.off) * ch + ci);
            if (j == 0) xv[it].x = v;
            if (j == 1) xv[it].y = v;
            if (j == 2) xv[it].z = v;
            if (j == 3) xv[it].w = v;
          }
        }
      }
    }
  }
}

// MODE 2 gather: this thread's row over the 8 voxels of each of its KG_T
// reduction groups (voxel table vt of the chunk)
__device__ __forceinline__ void gather2(float (&xw)[KG_T][8], const int2 *vt, int kgbase,
                                        int need_t, const float *src_t, int off_t, int xmask_t) {
#pragma unroll
  for (int g = 0; g < KG_T; ++g)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int2 e = vt[(kgbase + g) * 8 + j];
      xw[g][j] = (e.y & need_t) ? 0.f : __ldg(src_t + ((e.x + off_t) & xmask_t));
    }
}

// What 16 columns from c0 of an output row become as they are stored:
// forward: bias and ReLU; input gradient: NetGradEpi
template <int MODE>
__device__ __forceinline__ void epilogue16(float (&v)[16], const float *bias, int relu,
                                           const NetGradEpi &epi, size_t row, int N, int c0) {
  if (MODE == 0) {
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const float y = v[j] + (bias ? __ldg(bias + c0 + j) : 0.f);
      v[j] = relu && y < 0.f ? 0.f : y;
    }
    return;
  }
  const float4 *add =
      reinterpret_cast<const float4 *>(epi.add ? epi.add + row * epi.addp + c0 : nullptr);
  const float4 *mask =
      reinterpret_cast<const float4 *>(epi.mask ? epi.mask + row * N + c0 : nullptr);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    if (add) {
      const float4 w = __ldg(add + q);
      v[4 * q] = w.x + v[4 * q], v[4 * q + 1] = w.y + v[4 * q + 1];
      v[4 * q + 2] = w.z + v[4 * q + 2], v[4 * q + 3] = w.w + v[4 * q + 3];
    }
    if (mask) {
      const float4 w = __ldg(mask + q);
      v[4 * q] = w.x > 0.f ? v[4 * q] : 0.f;
      v[4 * q + 1] = w.y > 0.f ? v[4 * q + 1] : 0.f;
      v[4 * q + 2] = w.z > 0.f ? v[4 * q + 2] : 0.f;
      v[4 * q + 3] = w.w > 0.f ? v[4 * q + 3] : 0.f;
    }
  }
}

template <int MODE, int VEC>
__global__ void __launch_bounds__(TB_W, 3) k_conv_tc(TcArgs p) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint64_t bars[2];
  __shared__ uint32_t tbase;
  __shared__ TapEnt taps[81];     // MODE 0/1: the taps of the reduction
  __shared__ int ctap[16];        // MODE 1 at stride 2: the class's tap numbers
  __shared__ int2 rows_s[TB_M];   // MODE 0/1: row table (see below)
  __shared__ int2 vtab[3][TB_K];  // MODE 2: voxel tables of three chunks

  // tiles start on 1024-byte boundaries (128-byte swizzle)
  unsigned char *smem = smem_raw + ((1024u - (smem_addr(smem_raw) & 1023u)) & 1023u);
  const int tid = threadIdx.x, warp = tid >> 5;
  const int m0 = blockIdx.x * TB_M;
  const int N = p.N;
  const int nb = MODE == 2 ? 2 : 1;  // B tiles per stage
  const int stage_bytes = 2 * A_TILE + nb * N * TB_K * 2;
  const int rin = p.rin, rout = p.rout;
  // MODE 1 at stride 1 reads the output gradient like a forward pass with
  // mirrored taps.  At stride 2 an input voxel u = 2 w + par (per axis)
  // receives only the taps o with u + 1 - o even: o = 1 where par_a = 0, o
  // in {0, 2} where par_a = 1.  Block row blockIdx.y is the parity class par;
  // its rows are the voxels w of the output-gradient grid and its reduction
  // runs over its 1 to 16 taps, each reading w + (par + 1 - o) / 2.
  const bool cls = MODE == 1 && p.stride == 2;
  const int par = cls ? (int)blockIdx.y : 0;
  int ntap_c = 0;
  if (cls) {
    ntap_c = 1;
#pragma unroll
    for (int a = 0; a < 4; ++a) ntap_c *= 1 + ((par >> a) & 1);
  }
  const int Kc = cls ? ntap_c * p.cout : p.K;  // this block's reduction length
  const int kbeg = blockIdx.z * p.kslice;
  const int kend = min(Kc, kbeg + p.kslice);
  const int kpad_end = MODE == 0 ? min(p.Kpad, kbeg + p.kslice) : kend;
  const int nch = (kpad_end - kbeg + TB_K - 1) / TB_K;

  if (warp == 0) tmem_alloc(&tbase, (uint32_t)p.ncols);
  if (tid == 0) {
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
  }
  if (cls && tid < ntap_c) {
    // class tap tid: bit b of tid picks o = 0 or 2 on the b-th odd axis;
    // `need` marks the axes read at w + 1 (invalid where w + 1 = rout)
    int o[4], bit = 0, need = 0x100, off = 0, st = 1;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      if ((par >> a) & 1) {
        o[a] = ((tid >> bit) & 1) ? 2 : 0;
        ++bit;
      } else {
        o[a] = 1;
      }
      const int delta = (((par >> a) & 1) + 1 - o[a]) / 2;  // 0 or 1
      need |= delta << a;
      off += delta * st;
      st *= rout;
    }
    taps[tid] = TapEnt{need, off};
    ctap[tid] = o[0] + 3 * (o[1] + 3 * (o[2] + 3 * o[3]));
  }
  if ((MODE == 0 || (MODE == 1 && !cls)) && tid < 81) {
    // grid the taps read: the input (MODE 0) or the output gradient (MODE 1)
    const int e = MODE == 0 ? rin : rout;
    int o[4];
    tap_digits(tid, o);
    int need = 0x100, off = 0, st = 1;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int lo = MODE == 0 ? 0 : 2;  // the offset that falls off at coordinate 0
      need |= (o[a] == lo) << a;
      need |= (o[a] == 2 - lo) << (4 + a);
      off += (MODE == 0 ? o[a] - 1 : 1 - o[a]) * st;
      st *= e;
    }
    taps[tid] = TapEnt{need, off};
  }
  // row table: MODE 0: (input voxel of row * stride, edge mask);
  // MODE 1 at stride 1: (row's voxel, edge mask in the output-gradient grid);
  // MODE 1 at stride 2: (row's voxel w, bit a where w_a + 1 = rout)
  if ((MODE == 0 || MODE == 1) && tid < TB_M) {
    const int row = m0 + tid;
    int2 e = make_int2(0, 0x100);
    if (row < p.M) {
      const int ext = MODE == 0 || cls ? rout : rin;
      int c[4], v = row;
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        c[a] = v % ext;
        v /= ext;
      }
      if (MODE == 0) {
        int s[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) s[a] = c[a] * p.stride;
        e = make_int2(s[0] + rin * (s[1] + rin * (s[2] + rin * s[3])), edge_mask(s, rin));
      } else if (!cls) {
        e = make_int2(row, edge_mask(c, rout));
      } else {
        int m = 0;
#pragma unroll
        for (int a = 0; a < 4; ++a) m |= (c[a] + 1 >= rout) << a;
        e = make_int2(row, m);
      }
    }
    rows_s[tid] = e;
  }
  // MODE 2: this thread's row (tap, ci) reads src_t[(e.x + off_t) & xmask_t]
  // for each voxel e of the table that its `need` mask admits.  The bias
  // row, and rows past the end (never stored), read the constant 1.
  const int lrow = tid & (TB_M - 1), kgbase = (tid / TB_M) * KG_T;
  const int row2 = m0 + lrow;
  const float *src_t = &kOne;
  int need_t = 0x100, off_t = 0, xmask_t = 0;
  if (MODE == 2 && row2 < p.M - p.bias_row) {
    const int tap = row2 / p.cin;
    int o[4];
    tap_digits(tap, o);
    int st = 1, tapoff = 0;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      need_t |= (o[a] == 0) << a;
      need_t |= (o[a] == 2) << (4 + a);
      tapoff += (o[a] - 1) * st;
      st *= rin;
    }
    src_t = p.A;
    off_t = tapoff * p.cin + (row2 - tap * p.cin);
    xmask_t = -1;
  }
  if (MODE == 2) {
    fill_vtab(vtab[0], tid, kbeg, 0, nch, kend, rout, rin, p.stride, p.cin);
    fill_vtab(vtab[1], tid, kbeg, 1, nch, kend, rout, rin, p.stride, p.cin);
  }
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  // the tables above come from the arguments alone; from here on the operands
  // are read.  The next grid is let in when every block of this one holds its
  // tensor memory.
  pdl_wait();
  fence_before_sync();
  __syncthreads();
  pdl_launch_dependents();
  fence_after_sync();
  const uint32_t tacc = tbase;
  const uint32_t idesc = idesc_bf16_f32(TB_M, N);
  // MODE 0/1 staging: this thread loads 4 channels (half of reduction group
  // kgl) of rows rsub, rsub + 16, ..., so 16 lanes read 256 contiguous bytes
  // of a row when the chunk stays within one tap
  const int half = tid & 1, kgl = (tid >> 1) & 7, rsub = tid >> 4;
  const int ch = MODE == 0 ? p.cin : p.cout;

  // The next chunk's A values are loaded into registers right after this
  // chunk's are stored, so the loads are in flight across the barrier, the
  // MMA issue and the next stage's wait.
  float4 xv[TB_M / 16];  // MODE 0/1
  float xw[KG_T][8];     // MODE 2
  // warps 0-7 stage the operands; warp 8 only issues the MMAs, so that the
  // staging warps do not wait at the next barrier for the issuing thread
  const bool producer = tid < TB_T;
  if (producer) {
    if (MODE == 2)
      gather2(xw, vtab[0], kgbase, need_t, src_t, off_t, xmask_t);
    else
      gather01<VEC>(xv, p.A, kbeg + kgl * 8 + half * 4, Kc, taps, rows_s, rsub, ch);
  }

  int issued = 0;  // chunks whose MMAs were issued (block-uniform)
  bool bad = false;
  for (int i = 0; i < nch; ++i) {
    const int s = i & 1;
    const int k0 = kbeg + i * TB_K;
    unsigned char *st = smem + s * stage_bytes;
    unsigned char *Ahi = st, *Alo = st + A_TILE, *Bhi = st + 2 * A_TILE;
    unsigned char *Blo = Bhi + N * TB_K * 2;
    if (producer && i >= 2 && !mbar_wait_bounded(&bars[s], ((i - 2) >> 1) & 1)) bad = true;
    if (producer && !bad) {
      if (MODE == 2)
        fill_vtab(vtab[(i + 2) % 3], tid, kbeg, i + 2, nch, kend, rout, rin, p.stride, p.cin);
      // ---- A: store this chunk's registers
      if (MODE == 0 || MODE == 1) {
#pragma unroll
        for (int it = 0; it < TB_M / 16; ++it) {
          uint2 h, l;
          split4(xv[it], h, l);
          const uint32_t o = swz128(it * 16 + rsub, kgl) + half * 8;
          *reinterpret_cast<uint2 *>(Ahi + o) = h;
          *reinterpret_cast<uint2 *>(Alo + o) = l;
        }
      } else {
#pragma unroll
        for (int g = 0; g < KG_T; ++g) {
          uint4 h, l;
          split8(xw[g], h, l);
          const uint32_t o = swz128(lrow, kgbase + g);
          *reinterpret_cast<uint4 *>(Ahi + o) = h;
          *reinterpret_cast<uint4 *>(Alo + o) = l;
        }
      }
      // ---- B: N rows x 8 reduction groups
      for (int e = tid; e < N * 8; e += TB_T) {
        if (MODE == 2) {
          const int n = e % N, kg = e / N;
          float x[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int v = k0 + kg * 8 + j;
            x[j] = v < kend ? __ldg(p.B32 + (size_t)v * p.cout + n) : 0.f;
          }
          uint4 h, l;
          split8(x, h, l);
          const uint32_t o = swz128(n, kg);
          *reinterpret_cast<uint4 *>(Bhi + o) = h;
          *reinterpret_cast<uint4 *>(Blo + o) = l;
        } else {
          const int n = e >> 3, kg = e & 7;
          const int k = k0 + kg * 8;
          uint4 w = make_uint4(0, 0, 0, 0);
          if (MODE == 0) {
            w = __ldg(reinterpret_cast<const uint4 *>(p.Bw + (size_t)n * p.Kpad + k));
          } else if (k < Kc) {
            const int t = k / p.cout, c0 = k - t * p.cout;
            const int tap = cls ? ctap[t] : t;
            w = __ldg(reinterpret_cast<const uint4 *>(
                p.Bw + ((size_t)tap * p.cin + n) * p.cout + c0));
          }
          *reinterpret_cast<uint4 *>(Bhi + swz128(n, kg)) = w;
        }
      }
      // ---- A: the next chunk's loads
      if (i + 1 < nch) {
        if (MODE == 2)
          gather2(xw, vtab[(i + 1) % 3], kgbase, need_t, src_t, off_t, xmask_t);
        else
          gather01<VEC>(xv, p.A, k0 + TB_K + kgl * 8 + half * 4, Kc, taps, rows_s, rsub, ch);
      }
      fence_proxy_async_smem();
    }
    if (__syncthreads_or(bad)) break;
    if (tid == TB_T) {
      fence_after_sync();
      const uint32_t a_hi = smem_addr(Ahi), a_lo = smem_addr(Alo);
      const uint32_t b_hi = smem_addr(Bhi), b_lo = smem_addr(Blo);
#pragma unroll
      for (int kk = 0; kk < TB_K / 16; ++kk) {
        const uint64_t dah = smem_desc_sw128(a_hi + kk * 32);
        const uint64_t dal = smem_desc_sw128(a_lo + kk * 32);
        const uint64_t dbh = smem_desc_sw128(b_hi + kk * 32);
        mma_bf16(tacc, dah, dbh, idesc, (i | kk) != 0);
        mma_bf16(tacc, dal, dbh, idesc, 1);
        if (MODE == 2) mma_bf16(tacc, dah, smem_desc_sw128(b_lo + kk * 32), idesc, 1);
      }
      mma_commit(&bars[s]);
    }
    issued = i + 1;
  }

  // wait for the last issued chunk (its commit covers every earlier MMA)
  bool ok = !bad;
  if (issued > 0) {
    const int last = issued - 1;
    if (!mbar_wait_bounded(&bars[last & 1], (last >> 1) & 1)) ok = false;
  }
  if (!ok) *(volatile int *)p.err = FLOF_DEV_ERR_TC_TIMEOUT;
  ok = __syncthreads_and(ok);
  // a slice past this block's reduction (a parity class with fewer taps)
  // contributes zeros
  const bool empty = ok && issued == 0;
  ok = ok && issued > 0;
  fence_after_sync();
  if ((ok || empty) && producer) {
    // warp w reads tensor-memory lanes 32 (w % 4) .. + 31; warps 0-3 and
    // 4-7 take alternate 16-column groups
    const int q4 = warp & 3;
    const int r = m0 + 32 * q4 + (tid & 31);
    const bool split = MODE == 2 || gridDim.z > 1;
    // a slice holds every output row: M of them, or all rin^4 input voxels
    // of the parity classes
    const size_t rows_out = cls ? (size_t)rin * rin * rin * rin : (size_t)p.M;
    float *C = p.C + (split ? (size_t)blockIdx.z * rows_out * N : 0);
    // output row: the row itself, or for a parity class the input voxel
    // u = 2 w + par of the row's voxel w
    size_t orow = (size_t)r;
    if (cls && r < p.M) {
      int v = r, u = 0, mul = 1;
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        u += (2 * (v % rout) + ((par >> a) & 1)) * mul;
        v /= rout;
        mul *= rin;
      }
      orow = (size_t)u;
    }
    for (int c0 = 16 * (warp >> 2); c0 < N; c0 += 32) {
      float v[16];
      if (ok) {
        tmem_ld16(tacc + ((uint32_t)(32 * q4) << 16) + (uint32_t)c0, v);
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = 0.f;
      }
      if (r < p.M) {
        if (!split && MODE < 2) epilogue16<MODE>(v, p.bias, p.relu, p.epi, orow, N, c0);
        float4 *dst = reinterpret_cast<float4 *>(C + orow * N + c0);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          dst[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
      }
    }
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    fence_after_sync();
    tmem_dealloc(tacc, (uint32_t)p.ncols);
  }
}

// ---- stride-1 input gradient from a halo tile ------------------------------------
//
// out[v][n] = sum over taps and channels of A[v + 1 - tap][c] W[tap][n][c], 128
// output voxels per block: 8 along x times 16 rows.  Rows are counted through
// the plane padded by one voxel on each side, rho = z (R + 2) + y, so that
// the input row of tap (dy, dz) is row rho + dy + (R + 2) dz for every
// output row; the two rows between planes give results that are not stored.
// A chunk of the reduction is one t offset times 16 channels: the block loads
// the 16 + 2 + 2 (R + 2) rows of 10 voxels that its 27 (x, y, z) taps read,
// once, as BF16 parts hi and lo, in 16-byte units of 8 channels:
//   [part][channel group][row][10 voxels][16 bytes]
// Eight voxels along x of one channel group are then one core matrix of the
// unswizzled K-major operand wherever they start, so each tap is the same
// tile read from another start address: row groups 160 bytes apart, channel
// groups (rows x 160) bytes apart.  The im2col form of this file loads and
// converts every tap of every voxel anew: 81 values per input value instead
// of 3 (R + 2 + 9) 10 / 64 (13 at R = 16).  At the 16^4 network's layers
// (channels in the gradient -> columns): 16 -> 48 at 16^4 70 us (im2col 97),
// 32 -> 96 at 8^4 17 (36), 32 -> 32 at 8^4 11 (14), 64 -> 64 at 4^4 8 (15).
// Bound by the products' 128 x 16 operand reads and, at 4^4 and 8^4, by the
// latency of a chunk.
// The tensor core drops bits at each accumulation, so the products go to
// several accumulators that the stores add up in FP32: the lo parts to one,
// the hi parts of successive taps in turn to three (one where N > 64).  The
// forward pass keeps the im2col form: a change in the last bits of its
// activations moves some across zero, and with them the gradient.
struct HaloArgs {
  const float *A;          // output gradient, C channels
  const uint16_t *Bw;      // WB[tap][n][C]
  float *out;              // result rows x N, or slices of it
  int *err;
  int R, C, N, ncg;        // extent, channels, columns, groups of 16 channels
  int nx, nr;              // tiles along x, and of rows per plane
  int cslice;              // chunks per slice
  int pitch, nacc;         // accumulators: columns apart, number
  NetGradEpi epi;          // unsplit only
};

constexpr int HX = 10;     // voxels of a loaded row
constexpr int HTAPS = 27;  // taps of a chunk

__host__ __device__ constexpr int halo_rows(int R) { return 16 + 2 + 2 * (R + 2); }
__host__ __device__ constexpr int halo_stage(int R, int N) {
  return (halo_rows(R) * HX * 64 + HTAPS * 32 * N + 127) / 128 * 128;
}
__host__ __device__ constexpr int halo_table(int R) {
  return (halo_rows(R) * HX * 4 + 127) / 128 * 128;
}

__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_addr(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

__device__ __forceinline__ void load_ch8(float (&x)[8], const float *__restrict__ src) {
  const float4 a = __ldg(reinterpret_cast<const float4 *>(src));
  const float4 b = __ldg(reinterpret_cast<const float4 *>(src) + 1);
  x[0] = a.x, x[1] = a.y, x[2] = a.z, x[3] = a.w;
  x[4] = b.x, x[5] = b.y, x[6] = b.z, x[7] = b.w;
}

__global__ void __launch_bounds__(TB_W, 2) k_dgrad_halo(HaloArgs p) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint64_t bars[2];
  __shared__ uint32_t tbase;
  unsigned char *smem = smem_raw + ((128u - (smem_addr(smem_raw) & 127u)) & 127u);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int R = p.R, N = p.N, RP = R + 2;
  const int nv = halo_rows(R) * HX;  // voxels of a loaded slab
  int *voff = reinterpret_cast<int *>(smem);  // their offsets in a t plane, -1 outside
  unsigned char *stages = smem + halo_table(R);
  const int stage_bytes = halo_stage(R, N);

  const int tile = blockIdx.x;
  const int x0 = tile % p.nx * 8, rho0 = tile / p.nx % p.nr * 16, t = tile / (p.nx * p.nr);
  const int cbeg = blockIdx.z * p.cslice, cend = min(3 * p.ncg, cbeg + p.cslice);

  if (warp == 0) tmem_alloc(&tbase, (uint32_t)(p.pitch * p.nacc));
  if (tid == 0) {
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
  }
  for (int v = tid; v < nv; v += TB_W) {
    const int row = v / HX, rho = rho0 + row;
    const int x = x0 + (v - row * HX) - 1, z = rho / RP - 1, y = rho % RP - 1;
    const bool in = x >= 0 && x < R && y >= 0 && y < R && z >= 0 && z < R;
    voff[v] = in ? x + R * (y + R * z) : -1;
  }
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  // everything above comes from the arguments alone; the next grid is let in
  // when every block of this one holds its tensor memory
  pdl_wait();
  fence_before_sync();
  __syncthreads();
  pdl_launch_dependents();
  fence_after_sync();
  const uint32_t tacc = tbase;
  const uint32_t idesc = idesc_bf16_f32(TB_M, N);
  const bool producer = tid < TB_T;

  int issued = 0;  // chunks whose MMAs were issued (block-uniform)
  bool bad = false;
  for (int c = cbeg; c < cend; ++c) {
    const int dt = c / p.ncg, cg = c - dt * p.ncg, ti = t + dt - 1;
    if (ti < 0 || ti >= R) continue;  // the whole chunk falls off the grid
    const int s = issued & 1;
    unsigned char *Ahi = stages + s * stage_bytes, *Alo = Ahi + nv * 32, *Bs = Alo + nv * 32;
    if (producer && issued >= 2 && !mbar_wait_bounded(&bars[s], ((issued - 2) >> 1) & 1))
      bad = true;
    if (producer && !bad) {
      // ---- weights: 27 taps x 2 channel groups x N rows of 16 bytes
      for (int r = warp; r < HTAPS * 2; r += TB_T / 32) {
        const int tap = (r >> 1) + HTAPS * dt, c0 = cg * 16 + (r & 1) * 8;
        for (int n = lane; n < N; n += 32) {
          unsigned char *dst = Bs + (r * N + n) * 16;
          const uint16_t *src = p.Bw + ((size_t)(80 - tap) * N + n) * p.C + c0;
          cp_async16(dst, src);
        }
      }
      // ---- input slab: 2 channel groups x nv voxels, three at a time
      const float *base = p.A + (size_t)ti * R * R * R * p.C;
      constexpr int U = 3;
      for (int e0 = tid; e0 < 2 * nv; e0 += U * TB_T) {
        float x[U][8];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int e = e0 + u * TB_T;
          const int kg = e >= nv, v = e - kg * nv;
          const int off = e < 2 * nv ? voff[v] : -1;
#pragma unroll
          for (int j = 0; j < 8; ++j) x[u][j] = 0.f;
          if (off >= 0) load_ch8(x[u], base + (size_t)off * p.C + cg * 16 + kg * 8);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int e = e0 + u * TB_T;
          if (e < 2 * nv) {
            uint4 h, l;
            split8(x[u], h, l);
            *reinterpret_cast<uint4 *>(Ahi + e * 16) = h;
            *reinterpret_cast<uint4 *>(Alo + e * 16) = l;
          }
        }
      }
      cp_async_wait();
      fence_proxy_async_smem();
    }
    if (__syncthreads_or(bad)) break;
    if (tid == TB_T) {
      fence_after_sync();
      const uint32_t a_hi = smem_addr(Ahi), a_lo = smem_addr(Alo), b0 = smem_addr(Bs);
      const uint32_t lbo = (uint32_t)nv * 16;
      const int nhi = p.nacc - 1;
#pragma unroll 1
      for (int tap = 0, a = 0; tap < HTAPS; ++tap, a = a + 1 < nhi ? a + 1 : 0) {
        const int dz = tap / 9, dy = tap / 3 - dz * 3, dx = tap % 3;
        const uint32_t off = (uint32_t)(dx + HX * (dy + RP * dz)) * 16;
        const uint64_t db = smem_desc(b0 + tap * N * 32, (uint32_t)N * 16, 128);
        mma_bf16(tacc + (a + 1) * p.pitch, smem_desc(a_hi + off, lbo, HX * 16), db, idesc,
                 issued > 0 || tap >= nhi);
        mma_bf16(tacc, smem_desc(a_lo + off, lbo, HX * 16), db, idesc, (issued | tap) != 0);
      }
      mma_commit(&bars[s]);
    }
    ++issued;
  }

  // wait for the last issued chunk (its commit covers every earlier MMA)
  bool ok = !bad;
  if (issued > 0) {
    const int last = issued - 1;
    if (!mbar_wait_bounded(&bars[last & 1], (last >> 1) & 1)) ok = false;
  }
  if (!ok) *(volatile int *)p.err = FLOF_DEV_ERR_TC_TIMEOUT;
  ok = __syncthreads_and(ok);
  // a slice whose chunks all fall off the grid contributes zeros
  const bool empty = ok && issued == 0;
  ok = ok && issued > 0;
  fence_after_sync();
  if ((ok || empty) && producer) {
    const int q4 = warp & 3;
    const int r = 32 * q4 + lane;
    const int x = x0 + (r & 7), rho = rho0 + (r >> 3), z = rho / RP, y = rho - z * RP;
    const bool in = x < R && y < R && z < R;
    const size_t vol = (size_t)R * R * R;
    const bool split = gridDim.z > 1;
    const size_t orow = (size_t)t * vol + (in ? x + R * (y + R * z) : 0);
    float *out = p.out + (split ? (size_t)blockIdx.z * vol * R * N : 0);
    for (int c0 = 16 * (warp >> 2); c0 < N; c0 += 32) {
      float v[16];
      if (ok) {
        const uint32_t ta = tacc + ((uint32_t)(32 * q4) << 16) + (uint32_t)c0;
        tmem_ld16(ta + p.pitch, v);
        for (int k = 2; k <= p.nacc; ++k) {  // the others, the lo products last
          float w[16];
          tmem_ld16(ta + (k < p.nacc ? k : 0) * p.pitch, w);
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] += w[j];
        }
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = 0.f;
      }
      if (in) {
        if (!split) epilogue16<1>(v, nullptr, 0, p.epi, orow, N, c0);
        float4 *dst = reinterpret_cast<float4 *>(out + orow * N + c0);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          dst[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
      }
    }
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    fence_after_sync();
    tmem_dealloc(tacc, (uint32_t)(p.pitch * p.nacc));
  }
}

// ---- stride-1 weight gradient from halo tiles -----------------------------------
//
// grad[tap][ci][co] = sum over voxels u of in[u][ci] dout[u + 1 - tap][co].  A
// block keeps nine taps (all x and y offsets, one z and one t offset) of cc <=
// 64 input and 16 output channels in tensor memory and walks its share of the
// 128-voxel tiles (8 along x times 16 rows of the padded plane, as above).
// Both operands are stored in 16-byte units of 8 channels, voxel by voxel, one
// part (hi, lo) and channel group after another: the unswizzled MN-major
// layout, 8 voxels to a core matrix.  The 18 rows of 10 voxels of dout that the
// taps read are stored three times, each 8 voxels wide and shifted for its x
// offset, so that one MMA per y offset and 16 voxels multiplies (hi, lo) input
// channels (rows 0 .. cc - 1 and cc .. 2 cc - 1) by (hi, lo) x three x offsets
// x 16 output channels (96 columns), and a y offset is a start address one row
// on.  lo x lo is left out when the sums are taken out; rows past 2 cc multiply
// whatever follows in shared memory and are never read.  The tensor core drops
// bits at each accumulation: after at most WG_DRAIN tiles the sums are added to
// the block's slice in FP32 and begin anew (without, the network's gradient at
// 20^4 was 1.5 times as far from 64 bits as the im2col form's; with FP32 sums in
// registers the kernel spilled and took 80 us).  The bias gradient is summed
// in FP32 by the threads that stage dout, in the middle taps' block.
// Bound by the latency of a tile's loads (the 288 columns leave room for one
// block per SM): 48 -> 16 channels at 16^4 67 us (im2col 193; with the tap's
// shift on the input's side, one MMA of 32 columns per tap from a misaligned
// start, 120), 96 -> 32 at 8^4 25 (43), 64 -> 64 at 4^4 12 (12), 32 -> 32 at 8^4
// 14 (20).
struct WgradArgs {
  const float *in, *dout;
  float *out;             // slices: 2 per blockIdx.z, of 81 cin + 1 rows of cout
  int *err;
  int R, cin, cout;
  int cc, ncc, nco;       // input channels per block, blocks of them, of 16 output channels
  int nx, nr, tiles, per;  // tiles along x, of rows, in all, per slice
  int drain;              // tiles between drains
  FastDiv frp;            // by R + 2
};

constexpr int WG_CO = 16;                  // output channels of a block
constexpr int WG_ROWS = 18, WG_NV = WG_ROWS * HX;  // dout rows and voxels of a tile
constexpr int WG_BG = WG_ROWS * 128;       // bytes of a stored dout channel group
constexpr int WG_N = 6 * WG_CO;            // columns of an MMA
constexpr int WG_DRAIN = 20;               // most tiles (8 accumulations each) between drains
constexpr int WG_COLS = 512;               // tensor-memory columns: 3 WG_N, a power of two

__host__ __device__ constexpr int wg_stage(int cc) {
  return 2 * (cc / 8) * TB_M * 16 + 6 * (WG_CO / 8) * WG_BG;
}
// the MMA's 128 rows read 16 channel groups, whatever cc: room for the second
// stage's
__host__ __device__ constexpr int wg_smem(int cc) {
  const int st = wg_stage(cc), reach = st + 16 * TB_M * 16;
  return (2 * st > reach ? 2 * st : reach) + 128;
}

__global__ void __launch_bounds__(TB_W, 1) k_wgrad_halo(WgradArgs p) {
  constexpr int CO = WG_CO, NV = WG_NV, GO = CO / 8, BG = WG_BG;
  constexpr int UA = 4;                            // input units per thread (cc = 64)
  constexpr int UB = (GO * NV + TB_T - 1) / TB_T;  // dout units per thread
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint64_t bars[2];
  __shared__ uint32_t tbase;
  unsigned char *smem = smem_raw + ((128u - (smem_addr(smem_raw) & 127u)) & 127u);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int R = p.R, RP = R + 2, ga = p.cc / 8;
  const int stage_bytes = wg_stage(p.cc);
  // tap block (z offset, t offset), input and output channels
  int q = blockIdx.x;
  const int n0 = q % p.nco * CO;
  q /= p.nco;
  const int c0 = q % p.ncc * p.cc, tg = q / p.ncc;
  const int dz = tg % 3, dt = tg / 3;
  // the middle taps' block sees every voxel of dout
  const bool bias = dz == 1 && dt == 1 && c0 == 0;
  const int tbeg = blockIdx.z * p.per, tend = min(p.tiles, tbeg + p.per);

  if (warp == 0) tmem_alloc(&tbase, (uint32_t)WG_COLS);
  if (tid == 0) {
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
  }
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  pdl_wait();
  fence_before_sync();
  __syncthreads();
  pdl_launch_dependents();
  fence_after_sync();
  const uint32_t tacc = tbase;
  // both operands MN-major (bits 15 and 16)
  const uint32_t idesc = idesc_bf16_f32(TB_M, WG_N) | (1u << 15) | (1u << 16);
  const bool producer = tid < TB_T;

  float a[UA][8], b[UB][8], bsum[UB][8];
#pragma unroll
  for (int u = 0; u < UB; ++u)
#pragma unroll
    for (int j = 0; j < 8; ++j) bsum[u][j] = 0.f;
  // the loads of a tile: ga x 128 units of the input, GO x NV of dout
  auto load = [&](int tile) {
    const int x0 = tile % p.nx * 8, rho0 = tile / p.nx % p.nr * 16, t = tile / (p.nx * p.nr);
#pragma unroll
    for (int u = 0; u < UA; ++u) {
      const int e = tid + u * TB_T, g = e >> 7, r = e & (TB_M - 1);
      const int rho = rho0 + (r >> 3), z = (int)p.frp.div((uint32_t)rho);
      const int x = x0 + (r & 7), y = rho - z * RP;
#pragma unroll
      for (int j = 0; j < 8; ++j) a[u][j] = 0.f;
      if (g < ga && x < R && y < R && z < R)
        load_ch8(a[u], p.in + (size_t)(x + R * (y + R * (z + R * t))) * p.cin + c0 + g * 8);
    }
    const float *base = p.dout + (size_t)(t + 1 - dt) * R * R * R * p.cout + n0;
#pragma unroll
    for (int u = 0; u < UB; ++u) {
      const int e = tid + u * TB_T, g = e / NV, v = e - g * NV, row = v / HX;
      const int rho = rho0 + RP * (2 - dz) + row;
      const int zz = (int)p.frp.div((uint32_t)rho);
      const int x = x0 + (v - row * HX) - 1, y = rho - zz * RP - 1, z = zz - 1;
#pragma unroll
      for (int j = 0; j < 8; ++j) b[u][j] = 0.f;
      if (g < GO && x >= 0 && x < R && y >= 0 && y < R && z >= 0 && z < R)
        load_ch8(b[u], base + (size_t)(x + R * (y + R * z)) * p.cout + g * 8);
    }
  };
  // the sums in tensor memory, written (first) or added to the block's rows of
  // its slice; a hi row adds its products with lo dout.  Warps 0-3 and 4-7 take
  // alternate taps.
  const size_t slice = (size_t)(81 * p.cin + 1) * p.cout;
  float *out = p.out + 2 * (size_t)blockIdx.z * slice;
  auto drain = [&](bool first, bool zero) {
    const int r = 32 * (warp & 3) + lane, part = r >= p.cc, ci = r - part * p.cc;
    fence_after_sync();
#pragma unroll 1
    for (int tap = warp >> 2; tap < 9; tap += 2) {
      const uint32_t ta = tacc + ((uint32_t)(32 * (warp & 3)) << 16) +
                          (uint32_t)(tap / 3 * WG_N + tap % 3 * CO);
      float v[16], w[16];
      if (!zero) {
        tmem_ld16(ta, v);
        tmem_ld16(ta + 3 * CO, w);
      }
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = zero ? 0.f : part ? v[j] : v[j] + w[j];
      if (r < 2 * p.cc) {
        float4 *dst = reinterpret_cast<float4 *>(
            out + part * slice + (size_t)((tap + 9 * tg) * p.cin + c0 + ci) * p.cout + n0);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float4 o = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
          if (!first) {
            const float4 q4 = dst[j];
            o = make_float4(q4.x + o.x, q4.y + o.y, q4.z + o.z, q4.w + o.w);
          }
          dst[j] = o;
        }
      }
    }
    fence_before_sync();
  };
  // tiles whose dout tile falls off the grid in t contribute nothing
  const int plane = p.nx * p.nr;
  const int lo = max(tbeg, dt == 2 ? plane : 0);
  const int hi = min(tend, dt == 0 ? p.tiles - plane : p.tiles);

  int issued = 0;  // tiles whose MMAs were issued (block-uniform)
  bool bad = false, fresh = true;  // fresh: the next MMAs begin new sums
  if (producer && lo < hi) load(lo);
  for (int tile = lo; tile < hi; ++tile) {
    const int s = issued & 1;
    unsigned char *As = smem + s * stage_bytes, *Bs = As + 2 * ga * TB_M * 16;
    if (producer && issued >= 2 && !mbar_wait_bounded(&bars[s], ((issued - 2) >> 1) & 1))
      bad = true;
    if (tile != lo && (tile - lo) % p.drain == 0) {
      const int last = issued - 1;
      if (producer && !bad && !mbar_wait_bounded(&bars[last & 1], (last >> 1) & 1)) bad = true;
      if (producer && !bad) drain(issued == p.drain, false);
      fresh = true;
    }
    if (producer && !bad) {
#pragma unroll
      for (int u = 0; u < UA; ++u) {
        const int e = tid + u * TB_T;
        if ((e >> 7) < ga) {
          uint4 h, l;
          split8(a[u], h, l);
          *reinterpret_cast<uint4 *>(As + e * 16) = h;
          *reinterpret_cast<uint4 *>(As + (ga * TB_M + e) * 16) = l;
        }
      }
#pragma unroll
      for (int u = 0; u < UB; ++u) {
        const int e = tid + u * TB_T, g = e / NV, v = e - g * NV, row = v / HX;
        const int xx = v - row * HX;
        if (g < GO) {
          uint4 h, l;
          split8(b[u], h, l);
          // groups [part][x offset][channel group]; column x of the copy for
          // offset dx holds dout at x + 1 - dx, element x + 2 - dx of the row
#pragma unroll
          for (int dx = 0; dx < 3; ++dx) {
            const int x = xx - 2 + dx;
            if (x >= 0 && x < 8) {
              unsigned char *dst = Bs + (dx * GO + g) * BG + row * 128 + x * 16;
              *reinterpret_cast<uint4 *>(dst) = h;
              *reinterpret_cast<uint4 *>(dst + 3 * GO * BG) = l;
            }
          }
          // each voxel of dout once: the middle y offset's rows, eight columns
          if (bias && row >= 1 && row <= 16 && xx >= 1 && xx <= 8)
#pragma unroll
            for (int j = 0; j < 8; ++j) bsum[u][j] += b[u][j];
        }
      }
      if (tile + 1 < hi) load(tile + 1);  // in flight across the barrier and the MMAs
      fence_proxy_async_smem();
    }
    if (__syncthreads_or(bad)) break;
    if (tid == TB_T) {
      fence_after_sync();
      const uint32_t a0 = smem_addr(As), b0 = smem_addr(Bs);
#pragma unroll 1
      for (int ks = 0; ks < TB_M / 16; ++ks) {  // two rows of 8 voxels
        const uint64_t da = smem_desc(a0 + ks * 256, 128, TB_M * 16);
#pragma unroll
        for (int dy = 0; dy < 3; ++dy)
          mma_bf16(tacc + dy * WG_N, da, smem_desc(b0 + ks * 256 + (2 - dy) * 128, 128, BG), idesc,
                   !fresh || ks > 0);
      }
      mma_commit(&bars[s]);
    }
    fresh = false;
    ++issued;
  }

  // wait for the last issued tile (its commit covers every earlier MMA)
  bool ok = !bad;
  if (issued > 0) {
    const int last = issued - 1;
    if (!mbar_wait_bounded(&bars[last & 1], (last >> 1) & 1)) ok = false;
  }
  if (!ok) *(volatile int *)p.err = FLOF_DEV_ERR_TC_TIMEOUT;
  ok = __syncthreads_and(ok);
  // a slice without a tile: zeros
  if (ok && producer) drain(issued <= p.drain, issued == 0);
  if (bias) {
    // the threads' sums [group][voxel][8], then four partial sums per channel
    float *bs = reinterpret_cast<float *>(smem), *bp = bs + GO * NV * 8;
    if (producer)
#pragma unroll
      for (int u = 0; u < UB; ++u) {
        const int e = tid + u * TB_T;
        if (e < GO * NV)
#pragma unroll
          for (int j = 0; j < 8; ++j) bs[e * 8 + j] = bsum[u][j];
      }
    __syncthreads();
    if (tid < 4 * CO) {
      const int n = tid % CO, h = tid / CO;
      float x = 0.f;
      for (int v = h; v < NV; v += 4) x += bs[((n >> 3) * NV + v) * 8 + (n & 7)];
      bp[tid] = x;
    }
    __syncthreads();
    if (tid < 2 * CO) {
      const int n = tid % CO;
      const float x = (bp[n] + bp[CO + n]) + (bp[2 * CO + n] + bp[3 * CO + n]);
      out[(tid / CO) * slice + (size_t)81 * p.cin * p.cout + n0 + n] = tid < CO ? x : 0.f;
    }
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    fence_after_sync();
    tmem_dealloc(tacc, (uint32_t)WG_COLS);
  }
}

// What a sum of slices becomes as it is stored: forward: bias and ReLU; input
// gradient: NetGradEpi; weight gradient: added to what is there (acc).
struct SumEpi {
  const float *bias;
  int relu, acc;
  NetGradEpi grad;
};

// out[m][n] = sum over the slices + epilogue, four columns per thread.  GRP
// threads (of different warps) share an entry's slices, thread g adding g, g +
// GRP, ... in order, and thread 0 adds the GRP sums in order: with one thread
// per entry the two-channel layer's weight gradient (228 slices of 2608
// entries) was a chain of 228 loads, 6.4 us.  Forward sums, whose ReLU turns
// a last bit into a gradient's presence, are taken in slice order throughout.
template <int GRP>
__global__ void __launch_bounds__(256)
k_sum_slices(const float4 *__restrict__ work, float4 *out, uint32_t n4, int nz, FastDiv fN4,
             SumEpi e) {
  constexpr int NE = 256 / GRP;
  __shared__ float4 sh[GRP > 1 ? 256 : 1];
  const int lane = threadIdx.x % NE, g = threadIdx.x / NE;
  const uint32_t q = blockIdx.x * NE + lane;
  pdl_wait();
  pdl_launch_dependents();
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  if (q < n4) {
#pragma unroll 4
    for (int z = g; z < nz; z += GRP) {
      const float4 w = __ldg(work + (size_t)z * n4 + q);
      s.x += w.x, s.y += w.y, s.z += w.z, s.w += w.w;
    }
  }
  if (GRP > 1) {
    sh[threadIdx.x] = s;
    __syncthreads();
    if (g > 0) return;
    for (int k = 1; k < GRP; ++k) {
      const float4 w = sh[k * NE + lane];
      s.x += w.x, s.y += w.y, s.z += w.z, s.w += w.w;
    }
  }
  if (q >= n4) return;
  const uint32_t row = fN4.div(q), c = 4 * (q - row * fN4.d);
  if (e.bias) {
    const float *b = e.bias + c;
    s.x += __ldg(b), s.y += __ldg(b + 1), s.z += __ldg(b + 2), s.w += __ldg(b + 3);
  }
  if (e.relu) {
    s.x = s.x < 0.f ? 0.f : s.x, s.y = s.y < 0.f ? 0.f : s.y;
    s.z = s.z < 0.f ? 0.f : s.z, s.w = s.w < 0.f ? 0.f : s.w;
  }
  if (e.grad.add) {
    const float4 a = __ldg(
        reinterpret_cast<const float4 *>(e.grad.add + (size_t)row * e.grad.addp + c));
    s.x = a.x + s.x, s.y = a.y + s.y, s.z = a.z + s.z, s.w = a.w + s.w;
  }
  if (e.grad.mask) {
    const float4 y = __ldg(reinterpret_cast<const float4 *>(e.grad.mask) + q);
    s.x = y.x > 0.f ? s.x : 0.f, s.y = y.y > 0.f ? s.y : 0.f;
    s.z = y.z > 0.f ? s.z : 0.f, s.w = y.w > 0.f ? s.w : 0.f;
  }
  if (e.acc) {
    const float4 o = out[q];
    s.x = o.x + s.x, s.y = o.y + s.y, s.z = o.z + s.z, s.w = o.w + s.w;
  }
  out[q] = s;
}

// n entries of rows of N; every pointer and row length is a multiple of 16
// bytes (N is a multiple of 16, the network's tensors and layer offsets are)
void sum_slices(const float *work, float *out, long long n, int nz, int N, const SumEpi &e,
                cudaStream_t s) {
  const uint32_t n4 = (uint32_t)(n / 4);
  const FastDiv f((uint32_t)N / 4);
  if (nz >= 16 && !e.relu)
    launch_pdl(k_sum_slices<8>, (n4 + 31) / 32, 256, s, (const float4 *)work, (float4 *)out, n4,
               nz, f, e);
  else
    launch_pdl(k_sum_slices<1>, (n4 + 255) / 256, 256, s, (const float4 *)work, (float4 *)out, n4,
               nz, f, e);
}

// BF16 copies of one layer's weights W[tap][ci][co]: WB in the same order,
// WT[co][tap * cin + ci] with rows of length kpad (the tail stays zero).
// Both loops write consecutive entries from consecutive threads.
__global__ void k_weights_tc(const float *__restrict__ wq, uint16_t *__restrict__ wb,
                             uint16_t *__restrict__ wt, int taps, int cin, int cout, int kpad) {
  const long long K = (long long)taps * cin, n = K * cout;
  const long long step = (long long)gridDim.x * blockDim.x;
  auto bits = [](float x) {
    const __nv_bfloat16 b = __float2bfloat16_rn(x);
    return *reinterpret_cast<const uint16_t *>(&b);
  };
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += step)
    wb[q] = bits(wq[q]);
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += step) {
    const long long co = q / K, k = q - co * K;
    wt[(size_t)co * kpad + k] = bits(wq[(size_t)k * cout + co]);
  }
}

struct TcPlan {
  int nz, kslice;
};

// Slices of the reduction.  With `slots` = resident blocks per SM x SMs, a
// split into nz slices takes ceil(tiles nz / slots) waves of ceil(chunks /
// nz) chunks each, plus the pass that sums the slices: a launch (about 1.5
// chunk times) and reading nz M N floats (about 1.1 M of them per chunk
// time).  The split with the lowest estimate wins (at least four chunks per
// slice).
TcPlan tc_plan(long long M, long long K, int N, int resident) {
  const long long tiles = (M + TB_M - 1) / TB_M;
  const long long chunks = (K + TB_K - 1) / TB_K;
  const long long slots = (long long)std::max(resident, 1) * sm_count();
  const long long maxz = std::max(chunks / 4, 1LL);
  long long best = 1;
  double best_t = 1e300;
  for (long long nz = 1; nz <= maxz; ++nz) {
    const long long per = (chunks + nz - 1) / nz;
    const long long z = (chunks + per - 1) / per;  // slices actually used
    const long long waves = (tiles * z + slots - 1) / slots;
    const double t = (double)(waves * per) + (z > 1 ? 1.5 + (double)z * M * N / 1.1e6 : 0.0);
    if (t < best_t) best_t = t, best = z;
  }
  const long long per = (chunks + best - 1) / best;
  return TcPlan{(int)((chunks + per - 1) / per), (int)(per * TB_K)};
}

int pow2_cols(int n) {
  int c = 32;
  while (c < n) c <<= 1;
  return c;
}

template <int MODE>
int tc_smem(int N) {
  return 2 * (2 * A_TILE + (MODE == 2 ? 2 : 1) * N * TB_K * 2) + 1024;
}

// room for the largest stage pair (N = 128, two B tiles)
template <int MODE, int VEC>
void tc_attr() {
  fh::cuda_check(allow_smem<k_conv_tc<MODE, VEC>>(tc_smem<2>(128)),
                 "cudaFuncSetAttribute(k_conv_tc)");
}

// resident blocks per SM for N columns (N a multiple of 16 up to 128),
// queried once per shape
template <int MODE, int VEC>
int tc_resident(int N) {
  static std::atomic<int> cache[128 / 16 + 1];
  std::atomic<int> &slot = cache[N / 16];
  const int known = slot.load(std::memory_order_relaxed);
  if (known > 0) return known;
  tc_attr<MODE, VEC>();
  int nb = 0;
  fh::cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_conv_tc<MODE, VEC>, TB_W,
                                                               tc_smem<MODE>(N)),
                 "cudaOccupancyMaxActiveBlocksPerMultiprocessor(k_conv_tc)");
  nb = std::max(nb, 1);
  slot.store(nb, std::memory_order_relaxed);
  return nb;
}

template <int MODE, int VEC>
TcPlan tc_plan_for(long long M, long long K, int N) {
  return tc_plan(M, K, N, tc_resident<MODE, VEC>(N));
}

template <int MODE, int VEC>
void launch_tc(const TcArgs &a0, int nz, cudaStream_t s, int gy = 1) {
  TcArgs a = a0;
  a.ncols = pow2_cols(a.N);
  tc_attr<MODE, VEC>();
  dim3 grid((a.M + TB_M - 1) / TB_M, gy, nz);
  launch_pdl_smem(k_conv_tc<MODE, VEC>, grid, TB_W, tc_smem<MODE>(a.N), s, a);
  // a refused launch (configuration) is reported here, not by a later sync
  fh::cuda_check(cudaGetLastError(), "k_conv_tc launch");
}

// Slices of a stride-2 input gradient (16 parity classes of M rows, at most K
// = 16 cout reduction entries): enough blocks for about three per SM, at
// least two chunks per slice.
int cls_slices(long long M, long long K) {
  const long long blocks = (M + TB_M - 1) / TB_M * 16;
  const long long chunks = (K + TB_K - 1) / TB_K;
  long long nz = (3LL * sm_count() + blocks - 1) / blocks;
  nz = std::min(nz, std::max(chunks / 2, 1LL));
  const long long per = (chunks + nz - 1) / nz;
  return (int)((chunks + per - 1) / per);
}

// Halo tiles fit when two stages do (227 KB a block, a little of it static); nz slices of `cslice`
// chunks each.
struct HaloPlan {
  int nz, cslice, tiles, smem;
};
bool halo_ok(int R, int C, int N) {
  return C % 16 == 0 && halo_table(R) + 2 * halo_stage(R, N) + 128 <= 226 * 1024;
}

// A split into nz slices takes ceil(tiles nz / slots) waves of blocks, each
// about 3 us of set-up and stores and 1.3 us per chunk, plus the pass that
// sums the slices (2.5 us and 8 bytes per slice entry at 6 TB/s).
HaloPlan halo_plan(int R, int C, int N) {
  HaloPlan pl;
  pl.smem = halo_table(R) + 2 * halo_stage(R, N) + 128;
  pl.tiles = (R + 7) / 8 * ((R * (R + 2) + 15) / 16) * R;
  const int nch = 3 * (C / 16);
  const int resident = std::max(1, std::min(2, 228 * 1024 / (pl.smem + 1024)));
  const long long slots = (long long)resident * sm_count();
  const double sum_us = (double)R * R * R * R * N * 8 / 6e6;
  double best = 1e300;
  for (int nz = 1; nz <= nch; ++nz) {
    const int per = (nch + nz - 1) / nz, z = (nch + per - 1) / per;
    const long long waves = (pl.tiles * (long long)z + slots - 1) / slots;
    const double us = waves * (3.0 + 1.3 * per) + (z > 1 ? 2.5 + z * sum_us : 0.0);
    if (us < best) best = us, pl.nz = z, pl.cslice = per;
  }
  return pl;
}

void launch_halo(const HaloArgs &a0, const HaloPlan &pl, cudaStream_t s) {
  HaloArgs a = a0;
  a.pitch = pow2_cols(a.N);
  a.nacc = a.N > 64 ? 2 : 4;  // at most 256 columns: two blocks per SM
  a.ncg = a.C / 16;
  a.nx = (a.R + 7) / 8;
  a.nr = (a.R * (a.R + 2) + 15) / 16;
  a.cslice = pl.cslice;
  fh::cuda_check(allow_smem<k_dgrad_halo>(226 * 1024), "cudaFuncSetAttribute(k_dgrad_halo)");
  launch_pdl_smem(k_dgrad_halo, dim3(pl.tiles, 1, pl.nz), TB_W, (size_t)pl.smem, s, a);
  fh::cuda_check(cudaGetLastError(), "k_dgrad_halo launch");
}

// Weight gradient from halo tiles: blocks of at most 64 input and 16 output
// channels, tiles per slice.  A block takes about 4 us of set-up and stores and
// 1.2 us per tile, the sum of the slices 8 bytes per entry of a slice pair at 4
// TB/s; the count with the lowest estimate wins.
struct WgradPlan {
  int nz, per, tiles, ncc, nco;
  int blocks() const { return 9 * ncc * nco; }
};
WgradPlan wgrad_halo_plan(int R, int cin, int cout) {
  WgradPlan pl;
  pl.ncc = (cin + 63) / 64;
  while (cin % (8 * pl.ncc) != 0) ++pl.ncc;
  pl.nco = cout / 16;
  pl.tiles = (R + 7) / 8 * ((R * (R + 2) + 15) / 16) * R;
  const double sum_us = (81.0 * cin + 1) * cout * 8 / 4e6;
  double best = 1e300;
  const int most = std::min(pl.tiles, 64);
  for (int nz = 1; nz <= most; ++nz) {
    const int per = (pl.tiles + nz - 1) / nz, z = (pl.tiles + per - 1) / per;
    const int waves = (pl.blocks() * z + sm_count() - 1) / sm_count();
    const double us = waves * (4.0 + 1.2 * per) + z * sum_us;
    if (us < best) best = us, pl.nz = z, pl.per = per;
  }
  return pl;
}

// Halo tiles or im2col, by what each is expected to take.  Fitted to both over
// the four stride-1 layers' channels at extents 1 to 48 (halo against im2col, us,
// a layer at a time):
//   48 -> 16  8^4 13 / 19   16^4 67 / 193   48^4 4779 / 15127
//   32 -> 32  2^4 7.0 / 5.4  8^4 14 / 20    18^4 290 / 266    24^4 661 / 909
//   64 -> 64  3^4 10 / 8.4   8^4 28 / 37     9^4 72 / 46      12^4 147 / 141
// Tiles are 8 wide and a plane is padded, so a tile is mostly empty at an extent
// of 1 to 3 and half empty at 9; im2col packs its rows.  Where the
// estimates choose the slower form they lose up to 1.4 us (64 -> 64 at 5^4).
bool wgrad_halo_ok(int R, int cin, int cout, int stride) {
  if (stride != 1 || cin % 16 != 0 || cout % 16 != 0) return false;
  const WgradPlan pl = wgrad_halo_plan(R, cin, cout);
  const int waves = (pl.blocks() * pl.nz + sm_count() - 1) / sm_count();
  // a tile's loads, and the sums taken out every WG_DRAIN tiles
  const double tile = cin / pl.ncc < 64 ? 1.6 : 1.9;
  const double halo = 6.5 + waves * (tile * pl.per + 5.0 * ((pl.per - 1) / WG_DRAIN));
  const long long M = 81LL * cin + 1, K = (long long)R * R * R * R;
  const TcPlan tc = tc_plan_for<2, 0>(M, K, cout);
  // a chunk takes longer as blocks share an SM's loads
  const double share = (double)((M + TB_M - 1) / TB_M * tc.nz) / sm_count();
  const double chunk = (1.25 + 0.009 * cout) * std::max(1.0, 0.8 * share);
  const double sum = tc.nz > 1 ? 1.5 + (double)tc.nz * M * cout / 1.1e6 : 0.0;
  return halo <= 4.0 + chunk * (tc.kslice / TB_K) + sum;
}

void launch_wgrad_halo(const WgradArgs &a, const WgradPlan &pl, cudaStream_t s) {
  fh::cuda_check(allow_smem<k_wgrad_halo>(wg_smem(64)), "cudaFuncSetAttribute(k_wgrad_halo)");
  launch_pdl_smem(k_wgrad_halo, dim3(pl.blocks(), 1, pl.nz), TB_W, (size_t)wg_smem(a.cc), s, a);
  fh::cuda_check(cudaGetLastError(), "k_wgrad_halo launch");
}

TcPlan plan_fwd(long long M, long long K, int cin, int cout) {
  return cin % 8 == 0 ? tc_plan_for<0, 1>(M, K, cout) : tc_plan_for<0, 0>(M, K, cout);
}

}  // namespace

// ---- launchers --------------------------------------------------------------

int net_tc_kpad(int cin, int ks) {
  const int K = (ks == 3 ? 81 : 1) * cin;
  return (K + TB_K - 1) / TB_K * TB_K;
}

// the first layer has no input gradient
size_t net_tc_work(int rin, int rout, int cin, int cout, bool first) {
  size_t w = 0;
  const long long Vi = (long long)rin * rin * rin * rin, Vo = (long long)rout * rout * rout * rout;
  const bool same = rin == rout;
  const int nf = plan_fwd(Vo, net_tc_kpad(cin, 3), cin, cout).nz;
  if (nf > 1) w = std::max(w, (size_t)nf * (size_t)Vo * cout);
  if (!first) {
    const int nz = !same ? cls_slices(Vo, 16LL * cout)
                   : halo_ok(rin, cout, cin) ? halo_plan(rin, cout, cin).nz
                                       : tc_plan_for<1, 1>(Vi, 81LL * cout, cin).nz;
    if (nz > 1) w = std::max(w, (size_t)nz * (size_t)Vi * cin);
  }
  const int nw = wgrad_halo_ok(rin, cin, cout, same ? 1 : 2)
                     ? 2 * wgrad_halo_plan(rin, cin, cout).nz
                     : tc_plan_for<2, 0>(81LL * cin + 1, Vo, cout).nz;
  return std::max(w, (size_t)nw * (81 * cin + 1) * cout);
}

void net_weights_tc(const float *wq, uint16_t *wb, uint16_t *wt, int cin, int cout, int ks,
                    cudaStream_t s) {
  const int taps = ks == 3 ? 81 : 1;
  const long long n = (long long)taps * cin * cout;
  k_weights_tc<<<grid_for(n, 256), 256, 0, s>>>(wq, wb, wt, taps, cin, cout,
                                                net_tc_kpad(cin, ks));
}

void net_tc_conv_fwd(const float *in, const uint16_t *wt, const float *b, float *out,
                     float *work, int rin, int rout, int cin, int cout, int stride, int relu,
                     int *err, cudaStream_t s) {
  TcArgs a{};
  a.A = in;
  a.Bw = wt;
  a.err = err;
  a.rin = rin, a.rout = rout, a.cin = cin, a.cout = cout, a.stride = stride;
  a.M = rout * rout * rout * rout;
  a.N = cout;
  a.K = 81 * cin;
  a.Kpad = net_tc_kpad(cin, 3);
  a.relu = relu;
  const TcPlan pl = plan_fwd(a.M, a.Kpad, cin, cout);
  a.kslice = pl.kslice;
  a.bias = pl.nz > 1 ? nullptr : b;
  a.C = pl.nz > 1 ? work : out;
  if (cin % 8 == 0)
    launch_tc<0, 1>(a, pl.nz, s);
  else
    launch_tc<0, 0>(a, pl.nz, s);
  if (pl.nz > 1) {
    const long long n = (long long)a.M * a.N;
    sum_slices(work, out, n, pl.nz, a.N, SumEpi{b, relu, 0, {}}, s);
  }
}

void net_tc_conv_bwd_data(const float *dout, const uint16_t *wb, float *din, float *work,
                          int rin, int rout, int cin, int cout, int stride, NetGradEpi epi,
                          int *err, cudaStream_t s) {
  if (stride == 1 && halo_ok(rin, cout, cin)) {
    const HaloPlan pl = halo_plan(rin, cout, cin);
    HaloArgs a{};
    a.A = dout;
    a.Bw = wb;
    a.err = err;
    a.R = rin, a.C = cout, a.N = cin;
    a.epi = epi;
    a.out = pl.nz > 1 ? work : din;
    launch_halo(a, pl, s);
    if (pl.nz > 1)
      sum_slices(work, din, (long long)rin * rin * rin * rin * cin, pl.nz, cin,
                 SumEpi{nullptr, 0, 0, epi}, s);
    return;
  }
  TcArgs a{};
  a.epi = epi;
  a.A = dout;
  a.Bw = wb;
  a.err = err;
  a.rin = rin, a.rout = rout, a.cin = cin, a.cout = cout, a.stride = stride;
  a.N = cin;
  if (stride == 2) {
    // 16 parity classes of rout^4 rows each, at most 16 taps
    a.M = rout * rout * rout * rout;
    a.K = 16 * cout;
    a.Kpad = a.K;
    const int nz = cls_slices(a.M, a.K);
    const int chunks = (a.K + TB_K - 1) / TB_K;
    a.kslice = (chunks + nz - 1) / nz * TB_K;
    a.C = nz > 1 ? work : din;
    launch_tc<1, 1>(a, nz, s, 16);
    if (nz > 1) {
      const long long n = (long long)rin * rin * rin * rin * cin;
      sum_slices(work, din, n, nz, cin, SumEpi{nullptr, 0, 0, epi}, s);
    }
    return;
  }
  a.M = rin * rin * rin * rin;
  a.K = 81 * cout;
  a.Kpad = a.K;
  const TcPlan pl = tc_plan_for<1, 1>(a.M, a.K, a.N);
  a.kslice = pl.kslice;
  a.C = pl.nz > 1 ? work : din;
  launch_tc<1, 1>(a, pl.nz, s);
  if (pl.nz > 1) {
    const long long n = (long long)a.M * a.N;
    sum_slices(work, din, n, pl.nz, a.N, SumEpi{nullptr, 0, 0, epi}, s);
  }
}

void net_tc_conv_bwd_weight(const float *in, const float *dout, float *grad, float *work, int rin,
                            int rout, int cin, int cout, int stride, int acc, int *err,
                            cudaStream_t s) {
  if (wgrad_halo_ok(rin, cin, cout, stride)) {
    const WgradPlan pl = wgrad_halo_plan(rin, cin, cout);
    WgradArgs a{};
    a.in = in;
    a.dout = dout;
    a.out = work;
    a.err = err;
    a.R = rin, a.cin = cin, a.cout = cout;
    a.ncc = pl.ncc, a.cc = cin / pl.ncc, a.nco = pl.nco;
    a.nx = (rin + 7) / 8;
    a.nr = (rin * (rin + 2) + 15) / 16;
    a.tiles = pl.tiles, a.per = pl.per;
    const int drains = (pl.per + WG_DRAIN - 1) / WG_DRAIN;
    a.drain = (pl.per + drains - 1) / drains;
    a.frp = FastDiv((uint32_t)rin + 2);
    launch_wgrad_halo(a, pl, s);
    sum_slices(work, grad, (81LL * cin + 1) * cout, 2 * pl.nz, cout, SumEpi{nullptr, 0, acc, {}},
               s);
    return;
  }
  TcArgs a{};
  a.A = in;
  a.B32 = dout;
  a.err = err;
  a.rin = rin, a.rout = rout, a.cin = cin, a.cout = cout, a.stride = stride;
  a.M = 81 * cin + 1;  // the (tap, ci) rows and the bias row
  a.bias_row = 1;
  a.N = cout;
  a.K = rout * rout * rout * rout;
  a.Kpad = a.K;
  const TcPlan pl = tc_plan_for<2, 0>(a.M, a.K, a.N);
  a.kslice = pl.kslice;
  a.C = work;
  launch_tc<2, 0>(a, pl.nz, s);
  const long long n = (long long)a.M * a.N;
  sum_slices(work, grad, n, pl.nz, a.N, SumEpi{nullptr, 0, acc, {}}, s);
}

}  // namespace flof
