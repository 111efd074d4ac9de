// flof_cond.cu -- the steps either side of the solve: input conditioning of
// the 4D level sets (flof.py postProcessPhiData) and the output stage of the
// hi-res frames (flof.py time-SDF merge, blend union and writeResults
// smoothing).
//
// Reference:
//   repeatFrame4d          source/plugin/optflow4d.cpp:1254-1266
//   extrap4dLsSimple       source/plugin/optflow4d.cpp:1332-1406
//   knSimpleBlurSpecial    source/test.cpp:94-131
//   LevelsetGrid::join     source/levelset.cpp:114-118
//   Grid<T>::setBound      source/grid.cpp:462-473
//   Grid<T>::setBoundNeumann source/grid.cpp:475-511
//   knLoadPlaceGridIpol / knLoadPlaceGridRescale, shiftForwGrid4d
//                          source/plugin/optflow4d.cpp:1443-1458, 1596-1616
#include "flof_kernels.h"

namespace flof {

namespace {

constexpr int NT = 256;

// 3D cell of a linear index over an (X, Y, Z) box.
struct Box3 {
  FastDiv fx, fy;
  int ex, ey;
  __device__ __forceinline__ void decode(uint32_t n, int &i, int &j, int &k) const {
    const uint32_t q = fx.div(n);
    i = (int)(n - q * (uint32_t)ex);
    const uint32_t q2 = fy.div(q);
    j = (int)(q - q2 * (uint32_t)ey);
    k = (int)q2;
  }
};
Box3 box3(int ex, int ey) {
  Box3 b;
  b.fx = FastDiv((uint32_t)ex);
  b.fy = FastDiv((uint32_t)ey);
  b.ex = ex;
  b.ey = ey;
  return b;
}

// ---------------------------------------------------------------------------
// repeatFrame4d: every slice t in [t0, t1] of the bnd box gets the value
// interpolated at (i+.5, j+.5, k+.5, srct+.5).  The x, y, z coordinates
// land on cell centres, so each value depends on the cell itself at the two
// time slices around srct (the other corners carry weight zero).  The values
// are computed into a 3D buffer first and then written, so no thread reads a
// slice another thread is writing.
// ---------------------------------------------------------------------------
__global__ void k_repeat_frame_eval(const float *__restrict__ phi, Dims4 d, float srct,
                                    float *__restrict__ slice, Box3 bx, uint32_t n, int bnd) {
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    int i, j, k;
    bx.decode(q, i, j, k);
    i += bnd;
    j += bnd;
    k += bnd;
    slice[(idx_t)i + (idx_t)d.x * j + (idx_t)d.x * d.y * k] =
        interp4_real(phi, d, (float)i + 0.5f, (float)j + 0.5f, (float)k + 0.5f, srct + 0.5f);
  }
}

__global__ void k_repeat_frame_store(float *__restrict__ phi, Dims4 d,
                                     const float *__restrict__ slice, Box3 bx, uint32_t n,
                                     int bnd, int t0, int nt) {
  const idx_t sT = d.st();
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    int i, j, k;
    bx.decode(q, i, j, k);
    i += bnd;
    j += bnd;
    k += bnd;
    const idx_t id3 = (idx_t)i + (idx_t)d.x * j + (idx_t)d.x * d.y * k;
    const float v = slice[id3];
    for (int t = 0; t < nt; ++t) phi[id3 + (idx_t)(t0 + t) * sT] = v;
  }
}

// ---------------------------------------------------------------------------
// extrap4dLsSimple.  The reference marks cells 1 (inside the front), 2 (first
// layer), d+1 (filled by sweep d) in a Grid4d<int> and passes over the whole
// grid once per layer.  A sweep only needs to know which cells the last layer
// holds and which are reached, so both are kept as bit masks, one 32-bit word
// per 32 cells of an x row (1/32 of the int marks' bytes, and one word's
// neighbours tell about 32 cells): a lane forms the next layer's bits of its
// word from eleven words, and the warp then lists the new cells of its 32 words
// and evaluates them one per lane, so that a launch costs the masks plus the
// layer itself.
// A sweep reads phi only at the last layer's cells (final since the previous
// launch) and writes it only at newly reached ones, so sweeping in place has
// no read/write overlap.  At 48^3 x 72 a layer takes 6 to 7 us, launch and all
// (539 us for two calls of 40 layers), against 25 us for a pass over phi and int
// marks.
// ---------------------------------------------------------------------------
struct ExtrapShape {
  int X, Y, Z, T;
  int wpr;             // words per x row
  uint32_t nwords;     // wpr * Y * Z * T
  FastDiv fw, fy, fz;  // word index -> row, row -> (y, z, t)
  uint32_t nin;        // words of the inner rows
  FastDiv gy, gz;      // inner row -> (y - 1, z - 1, t - 1)
};

// the inner cells (1 <= x < X-1) among the 32 of word wx
__device__ __forceinline__ unsigned inner_bits(const ExtrapShape &e, int wx) {
  const int lo = 32 * wx, hi = e.X - 1 - lo;  // bits below hi
  unsigned m = hi >= 32 ? 0xffffffffu : hi > 0 ? (1u << hi) - 1u : 0u;
  if (wx == 0) m &= ~1u;
  return m;
}
__device__ __forceinline__ void word_row(const ExtrapShape &e, uint32_t w, uint32_t &row, int &wx,
                                         bool &inner) {
  row = e.fw.div(w);
  wx = (int)(w - row * (uint32_t)e.wpr);
  const uint32_t r2 = e.fy.div(row), t = e.fz.div(r2);
  const int y = (int)(row - r2 * (uint32_t)e.Y), z = (int)(r2 - t * (uint32_t)e.Z);
  inner = y >= 1 && y < e.Y - 1 && z >= 1 && z < e.Z - 1 && (int)t >= 1 && (int)t < e.T - 1;
}

// the cells inside the front, one warp per word
__global__ void k_extrap_mark(const float *__restrict__ phi, unsigned *__restrict__ front,
                              unsigned *__restrict__ next, unsigned *__restrict__ seen, ExtrapShape e,
                              int inside) {
  pdl_wait();
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31;
  const uint32_t nwarps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < e.nwords; w += nwarps) {
    uint32_t row;
    int wx;
    bool inner;
    word_row(e, w, row, wx, inner);
    bool in = false;
    if (inner && (inner_bits(e, wx) >> lane & 1u)) {
      const float v = __ldg(phi + (idx_t)row * e.X + 32 * wx + lane);
      in = inside ? v > 0.f : v < 0.f;
    }
    const unsigned bits = __ballot_sync(0xffffffffu, in);
    if (lane == 0) {
      front[w] = bits;
      seen[w] = bits;
      next[w] = 0;  // the steps write the inner rows only
    }
  }
}

// One layer: next = the unreached inner neighbours of `front`.  EVAL: each
// gets the mean of its neighbours in `front`, added in nbs4d's order
// (optflow4d.cpp:1323-1326: -x,+x,-y,+y,-z,+z,-t,+t), plus direction; the
// first layer keeps its values.  An empty front costs a launch as in the
// reference: a flag to end early, stored by each warp with new cells, took
// ten times the layer's own time (thousands of stores to one address).
template <bool EVAL>
__global__ void __launch_bounds__(128, 16)
k_extrap_step(float *__restrict__ phi, const unsigned *__restrict__ front,
              unsigned *__restrict__ next, unsigned *__restrict__ seen, ExtrapShape e, float direction) {
  __shared__ uint16_t list[4][1024];
  pdl_wait();
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31;
  const uint32_t q0 = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t sy = (uint32_t)e.wpr, sz = sy * e.Y, st = sz * e.Z;
  unsigned f = 0, fl = 0, fr = 0, ym = 0, yp = 0, zm = 0, zp = 0, tm = 0, tp = 0, nw = 0;
  uint32_t row = 0;
  int wx = 0;
  if (q0 < e.nin) {
    const uint32_t r = e.fw.div(q0), r2 = e.gy.div(r), t = e.gz.div(r2);
    wx = (int)(q0 - r * sy);
    const uint32_t y = 1 + r - r2 * e.gy.d, z = 1 + r2 - t * e.gz.d;
    row = y + (uint32_t)e.Y * (z + (uint32_t)e.Z * (1 + t));
    const uint32_t w = row * sy + wx;
    const unsigned s = seen[w];
    f = __ldg(front + w);
    if (wx > 0) fl = __ldg(front + w - 1) >> 31;
    if (wx + 1 < e.wpr) fr = __ldg(front + w + 1) << 31;
    ym = __ldg(front + w - sy);
    yp = __ldg(front + w + sy);
    zm = __ldg(front + w - sz);
    zp = __ldg(front + w + sz);
    tm = __ldg(front + w - st);
    tp = __ldg(front + w + st);
    nw = ((f << 1) | fl | (f >> 1) | fr | ym | yp | zm | zp | tm | tp) & ~s & inner_bits(e, wx);
    if (nw) seen[w] = s | nw;
    next[w] = nw;
  }
  const unsigned all = 0xffffffffu;
  if (!EVAL || !__any_sync(all, nw != 0)) return;
  // the warp's new cells as a list, (lane of the word) * 32 + bit
  uint16_t *const mine = list[threadIdx.x >> 5];
  const int cnt = __popc(nw);
  int pos = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(all, pos, o);
    if (lane >= o) pos += v;
  }
  const int total = __shfl_sync(all, pos, 31);
  pos -= cnt;
  for (unsigned b = nw; b; b &= b - 1) mine[pos++] = (uint16_t)(lane * 32 + __ffs(b) - 1);
  __syncwarp();
  // the front at the -x and +x neighbours of each cell of the word
  const unsigned xm = (f << 1) | fl, xp = (f >> 1) | fr;
  const idx_t sY = e.X, sZ = sY * e.Y, sT = sZ * e.Z;
  const idx_t base = (idx_t)row * e.X + 32 * wx;
  for (int q = 0; q < total; q += 32) {
    const bool live = q + lane < total;
    const int ent = live ? mine[q + lane] : 0;
    const int src = ent >> 5, bit = ent & 31;
    const unsigned hit[8] = {__shfl_sync(all, xm, src), __shfl_sync(all, xp, src),
                             __shfl_sync(all, ym, src), __shfl_sync(all, yp, src),
                             __shfl_sync(all, zm, src), __shfl_sync(all, zp, src),
                             __shfl_sync(all, tm, src), __shfl_sync(all, tp, src)};
    const idx_t id = __shfl_sync(all, base, src) + bit;
    if (live) {
      const idx_t off[8] = {-1, 1, -sY, sY, -sZ, sZ, -sT, sT};
      float v[8];
#pragma unroll
      for (int m = 0; m < 8; ++m) v[m] = (hit[m] >> bit & 1u) ? phi[id + off[m]] : 0.f;
      int nbs = 0;
      float avg = 0.f;
#pragma unroll
      for (int m = 0; m < 8; ++m)
        if (hit[m] >> bit & 1u) {
          avg += v[m];
          nbs++;
        }
      phi[id] = avg / (float)nbs + direction;
    }
  }
}

// inner cells that no layer reached, one warp per word
__global__ void k_extrap_remaining(float *__restrict__ phi, const unsigned *__restrict__ seen,
                                   ExtrapShape e, float value) {
  pdl_wait();
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31;
  const uint32_t nwarps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < e.nwords; w += nwarps) {
    uint32_t row;
    int wx;
    bool inner;
    word_row(e, w, row, wx, inner);
    if (!inner) continue;
    const unsigned left = inner_bits(e, wx) & ~__ldg(seen + w);
    if (left >> lane & 1u) phi[(idx_t)row * e.X + 32 * wx + lane] = value;
  }
}

// ---------------------------------------------------------------------------
// knSimpleBlurSpecial over the bnd = 1 box of a 3D grid (k = 0 only for a 2D
// grid): cells outside isInBounds(bord) or below thresh are copied, the rest
// get the mean of their 6 (3D) or 4 (2D) face neighbours, added in the
// reference's order and scaled by the double constant 1/6 (1/4).  The ring
// outside the box is not written.
// ---------------------------------------------------------------------------
__global__ void k_simple_blur_special(const float *__restrict__ a, float *__restrict__ tmp,
                                      int X, int Y, int Z, Box3 bx, uint32_t n, float thresh,
                                      int bord) {
  const bool is3d = Z > 1;
  const idx_t sY = X, sZ = (idx_t)X * Y;
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    int i, j, k;
    bx.decode(q, i, j, k);
    i += 1;
    j += 1;
    if (is3d) k += 1;
    const idx_t id = (idx_t)i + sY * j + sZ * k;
    bool inb = i >= bord && j >= bord && i < X - bord && j < Y - bord;
    inb = inb && (is3d ? (k >= bord && k < Z - bord) : (k == 0));
    const float v = a[id];
    if (!inb || v < thresh) {
      tmp[id] = v;
      continue;
    }
    float s = a[id + 1] + a[id - 1];
    s = s + a[id + sY];
    s = s + a[id - sY];
    if (is3d) {
      s += a[id + sZ] + a[id - sZ];
      tmp[id] = (float)((double)s * (1. / 6.));
    } else {
      tmp[id] = (float)((double)s * (1. / 4.));
    }
  }
}

// LevelsetGrid::join: a = std::min(a, b), i.e. b only where b < a.
__global__ void k_join(float *__restrict__ a, const float *__restrict__ b, long long n) {
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
       q += (long long)gridDim.x * blockDim.x) {
    const float x = a[q], y = b[q];
    a[q] = (y < x) ? y : x;
  }
}

// Grid<T>::setBound for a 3D (or 2D, Z == 1) grid: every cell with
// i <= w, i >= X-1-w, j <= w, j >= Y-1-w or, in 3D, the same in k.
__global__ void k_set_bound3(float *__restrict__ a, int X, int Y, int Z, int nc, float4 v,
                             int w, Box3 bx, uint32_t n) {
  const bool is3d = Z > 1;
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    int i, j, k;
    bx.decode(q, i, j, k);
    const bool b = i <= w || i >= X - 1 - w || j <= w || j >= Y - 1 - w ||
                   (is3d && (k <= w || k >= Z - 1 - w));
    if (!b) continue;
    if (nc == 4)
      ((float4 *)a)[q] = v;
    else
      a[q] = v.x;
  }
}

// Grid<T>::setBoundNeumann for a 3D (or 2D) grid: boundary cells copy the
// nearest cell just inside the w+1 wide ring.  The cells read are never
// boundary cells, so the kernel runs in place.
__global__ void k_set_bound_neumann3(float *__restrict__ a, int X, int Y, int Z, int nc, int w,
                                     Box3 bx, uint32_t n) {
  const bool is3d = Z > 1;
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    int i, j, k;
    bx.decode(q, i, j, k);
    bool set = false;
    int si = i, sj = j, sk = k;
    if (i <= w) { si = w + 1; set = true; }
    if (i >= X - 1 - w) { si = X - 1 - w - 1; set = true; }
    if (j <= w) { sj = w + 1; set = true; }
    if (j >= Y - 1 - w) { sj = Y - 1 - w - 1; set = true; }
    if (is3d) {
      if (k <= w) { sk = w + 1; set = true; }
      if (k >= Z - 1 - w) { sk = Z - 1 - w - 1; set = true; }
    }
    if (!set) continue;
    const idx_t src = (idx_t)si + (idx_t)X * sj + (idx_t)X * Y * sk;
    if (nc == 4)
      ((float4 *)a)[q] = ((const float4 *)a)[src];
    else
      a[q] = a[src];
  }
}

// knLoadPlaceGridIpol: phi(i,j,k,slice) += wc * trilinear(src3, ijk * sf + off)
// over the bnd = 1 box of phi's (x,y,z) extent.
__global__ void k_place_slice(float *__restrict__ phi, Dims4 d, int slice,
                              const float *__restrict__ src, int sx, int sy, int sz, float3 sf,
                              float3 off, float wc, Box3 bx, uint32_t n) {
  const int size[3] = {sx, sy, sz};
  const idx_t sZs = sz > 1 ? (idx_t)sx * sy : 0;  // a 2D grid has no z stride
  const idx_t base = (idx_t)slice * d.st();
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    int i, j, k;
    bx.decode(q, i, j, k);
    i += 1;
    j += 1;
    k += 1;
    const float p0 = (float)i * sf.x + off.x;
    const float p1 = (float)j * sf.y + off.y;
    const float p2 = (float)k * sf.z + off.z;
    const float v = interp3_real(src, size, sZs, p0, p1, p2);
    const idx_t id = base + (idx_t)i + (idx_t)d.x * j + d.sz() * k;
    phi[id] += wc * v;
  }
}

// tmp(i,j,k) += v over the bnd = 1 box of a 3D grid (the sdfIsoOff fix-up of
// loadPlaceGrid4d, optflow4d.cpp:1566-1572).
__global__ void k_add_inner3(float *__restrict__ a, int X, int Y, int Z, float v, Box3 bx,
                             uint32_t n) {
  const bool is3d = Z > 1;
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    int i, j, k;
    bx.decode(q, i, j, k);
    i += 1;
    j += 1;
    if (is3d) k += 1;
    a[(idx_t)i + (idx_t)X * j + (idx_t)X * Y * k] += v;
  }
}

// knLoadPlaceGridRescale: phi(i,j,k,t) *= w[t] where w[t] > 0, bnd = 1 box.
__global__ void k_rescale_slices(float *__restrict__ phi, Dims4 d, const float *__restrict__ w,
                                 BoxDecoder bx, uint32_t n) {
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    int i, j, k, t;
    bx.decode(q, i, j, k, t);
    const float wt = w[t];
    if (wt <= 0.f) continue;
    const idx_t id = d.index(i, j, k, t);
    phi[id] *= wt;
  }
}

}  // namespace

void launch_repeat_frame(float *phi, Dims4 d, float srct, int t0, int t1, int bnd, float *slice,
                         cudaStream_t s) {
  const int ex = d.x - 2 * bnd, ey = d.y - 2 * bnd, ez = d.z - 2 * bnd;
  if (ex <= 0 || ey <= 0 || ez <= 0 || t1 < t0) return;
  const uint32_t n = (uint32_t)((long long)ex * ey * ez);
  const Box3 bx = box3(ex, ey);
  k_repeat_frame_eval<<<grid_for(n, NT), NT, 0, s>>>(phi, d, srct, slice, bx, n, bnd);
  k_repeat_frame_store<<<grid_for(n, NT), NT, 0, s>>>(phi, d, slice, bx, n, bnd, t0,
                                                      t1 - t0 + 1);
}

static uint32_t extrap_nwords(Dims4 d) {
  return (uint32_t)((long long)((d.x + 31) / 32) * d.y * d.z * d.t);
}
size_t extrap_scratch_bytes(Dims4 d) { return (size_t)extrap_nwords(d) * 12; }

void launch_extrap(float *phi, Dims4 d, int distance, int inside, void *scratch, cudaStream_t s) {
  ExtrapShape e;
  e.X = d.x;
  e.Y = d.y;
  e.Z = d.z;
  e.T = d.t;
  e.wpr = (d.x + 31) / 32;
  e.nwords = extrap_nwords(d);
  e.fw = FastDiv((uint32_t)e.wpr);
  e.fy = FastDiv((uint32_t)d.y);
  e.fz = FastDiv((uint32_t)d.z);
  e.nin = (uint32_t)((long long)e.wpr * (d.y - 2) * (d.z - 2) * (d.t - 2));
  e.gy = FastDiv((uint32_t)(d.y - 2));
  e.gz = FastDiv((uint32_t)(d.z - 2));
  unsigned *front = (unsigned *)scratch, *next = front + e.nwords, *seen = next + e.nwords;
  const float direction = inside ? -1.f : 1.f;
  const unsigned gw = (unsigned)grid_for((long long)e.nwords * 32, NT);
  const unsigned gs = (e.nin + 127) / 128;
  launch_pdl(k_extrap_mark, gw, NT, s, (const float *)phi, front, next, seen, e,
             inside);
  launch_pdl(k_extrap_step<false>, gs, 128, s, phi, (const unsigned *)front, next, seen, e,
             direction);
  for (int dd = 2; dd < 1 + distance; ++dd) {
    unsigned *sw = front;
    front = next;
    next = sw;
    launch_pdl(k_extrap_step<true>, gs, 128, s, phi, (const unsigned *)front, next, seen, e,
               direction);
  }
  launch_pdl(k_extrap_remaining, gw, NT, s, phi, (const unsigned *)seen, e,
             direction * (float)(distance + 2));
}

void launch_simple_blur_special(const float *a, float *tmp, int X, int Y, int Z, float thresh,
                                int bord, cudaStream_t s) {
  const int ex = X - 2, ey = Y - 2, ez = Z > 1 ? Z - 2 : 1;
  if (ex <= 0 || ey <= 0 || ez <= 0) return;
  const uint32_t n = (uint32_t)((long long)ex * ey * ez);
  k_simple_blur_special<<<grid_for(n, NT), NT, 0, s>>>(a, tmp, X, Y, Z, box3(ex, ey), n, thresh,
                                                       bord);
}

void launch_join(float *a, const float *b, long long n, cudaStream_t s) {
  k_join<<<grid_for(n, NT), NT, 0, s>>>(a, b, n);
}

void launch_set_bound3(float *a, int X, int Y, int Z, int nc, float4 v, int w, cudaStream_t s) {
  const uint32_t n = (uint32_t)((long long)X * Y * Z);
  k_set_bound3<<<grid_for(n, NT), NT, 0, s>>>(a, X, Y, Z, nc, v, w, box3(X, Y), n);
}

void launch_set_bound_neumann3(float *a, int X, int Y, int Z, int nc, int w, cudaStream_t s) {
  const uint32_t n = (uint32_t)((long long)X * Y * Z);
  k_set_bound_neumann3<<<grid_for(n, NT), NT, 0, s>>>(a, X, Y, Z, nc, w, box3(X, Y), n);
}

void launch_place_slice(float *phi, Dims4 d, int slice, const float *src, const int sdims[3],
                        const float sf[3], const float off[3], float wc, cudaStream_t s) {
  const int ex = d.x - 2, ey = d.y - 2, ez = d.z - 2;
  if (ex <= 0 || ey <= 0 || ez <= 0) return;
  const uint32_t n = (uint32_t)((long long)ex * ey * ez);
  k_place_slice<<<grid_for(n, NT), NT, 0, s>>>(phi, d, slice, src, sdims[0], sdims[1], sdims[2],
                                               make_float3(sf[0], sf[1], sf[2]),
                                               make_float3(off[0], off[1], off[2]), wc,
                                               box3(ex, ey), n);
}

void launch_add_inner3(float *a, int X, int Y, int Z, float v, cudaStream_t s) {
  const int ex = X - 2, ey = Y - 2, ez = Z > 1 ? Z - 2 : 1;
  if (ex <= 0 || ey <= 0 || ez <= 0) return;
  const uint32_t n = (uint32_t)((long long)ex * ey * ez);
  k_add_inner3<<<grid_for(n, NT), NT, 0, s>>>(a, X, Y, Z, v, box3(ex, ey), n);
}

void launch_rescale_slices(float *phi, Dims4 d, const float *w, cudaStream_t s) {
  if (d.x < 3 || d.y < 3 || d.z < 3 || d.t < 3) return;
  const uint32_t n = (uint32_t)((long long)(d.x - 2) * (d.y - 2) * (d.z - 2) * (d.t - 2));
  k_rescale_slices<<<grid_for(n, NT), NT, 0, s>>>(
      phi, d, w, make_decoder(d.x - 2, d.y - 2, d.z - 2, 1, 1, 1, 1), n);
}

}  // namespace flof
