// flof_resident.cu -- the Jacobi-PCG of a small level as one cooperative
// launch (GridCGOptflow4d::solve, optflow4d.cpp:268-329: the same iteration
// and stop rule as the chained kernels of flof_solve.cu).
//
// A level of up to a few million cells fits in L2, and its chained iteration
// (matvec, update, direction) is bound by the three kernel boundaries and
// their last-block sums, not by its bytes.  Here one block per SM keeps its
// contiguous run of interior cells for the whole solve: the residual (and for
// the smaller levels the gradient) stays in shared memory and A p in
// registers; only p, which the neighbours read, and x pass through L1 and L2.
// An iteration has two grid barriers:
//   phase 1  q = A p and three dot products, p.q, q.z and q.M^-1 q
//   barrier  every block sums the blocks' partials in the same order, so all
//            compute the same alpha and beta
//   phase 2  r -= alpha q, x += alpha p, p = z + beta p, z.r and max r
//   barrier  p is visible; z.r and max r are read after the next phase 1
// beta needs the next z.r before r is updated; with r' = r - a q it is
//   z'.r' = z.r - 2 a q.z + a^2 q.M^-1 q,
// formed in double from this iteration's sums for this beta only; the next
// alpha uses z.r summed afresh from the updated r, so nothing accumulates.
// The stop rule is read one phase later than in the chained kernels: the
// phase 1 run past the last update is not used.
//
// Time per iteration on GB300 (100 iterations, chained kernels / this):
//   12^3 x 8    6000 cells   15.6 / 6.2 us      32^4       810k   38 / 20 us
//   16^4          38k        17.0 / 7.2 us      45x38x41x30 1.7M  68 / 47 us
//   24^3 x 16    149k        22.6 / 9.2 us
//
// The blocks wait on one another, so the launch is cooperative and the blocks
// of all launches in flight are counted (ResidentShare): they never exceed
// the SMs.  Other work on the device can still keep a block from starting for
// as long as it runs (a caller's long kernel on another stream).  So the first
// meeting of the blocks is a gate (grid_gate): either all of them are there
// within its wait and go on, or they leave the level as they found it, for the
// chained kernels.  Past the gate every block is resident; the barriers' waits
// are bounded all the same, and a block that gives up there records
// FLOF_DEV_ERR_GRID_TIMEOUT and returns, and the others after it.
//
// The sums are formed per work group of `per` cells and then over the groups
// in order, and a block holds M groups, so the result does not depend on M:
// one solve alone spreads its groups over the SMs (M = 1), the solves of a
// batch take a quarter of the SMs each (M = 4) and run side by side.
#include "flof_kernels.h"

namespace flof {

namespace {

constexpr int GRID_WAIT_LIMIT = 1 << 22;  // polls (about half a microsecond each)

// Jacobi preconditioner of a row (as in flof_solve.cu)
__device__ __forceinline__ float4 res_precond(const float4 g, float diag) {
  float4 p;
  p.x = __frcp_rn(g.x * g.x + diag);
  p.y = __frcp_rn(g.y * g.y + diag);
  p.z = __frcp_rn(g.z * g.z + diag);
  p.w = __frcp_rn(g.w * g.w + diag);
  return p;
}

// All blocks' writes before the barrier are visible to all blocks after it;
// false when the others did not arrive in time.
__device__ __forceinline__ bool grid_barrier(unsigned int *counter, unsigned int target,
                                             int *ok_sh) {
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
    int ok = 0;
    for (int n = 0; n < GRID_WAIT_LIMIT; ++n) {
      unsigned int v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
      if ((int)(v - target) >= 0) {
        ok = 1;
        break;
      }
    }
    *ok_sh = ok;
  }
  __syncthreads();
  return *ok_sh != 0;
}

// The first meeting: true when every block has come.  The last one to come
// opens the gate; a block whose wait ends first shuts it.  Whichever happens
// first holds for all blocks, those that start later among them.  The block
// that shuts it tells the host.  limit: polls to wait; 0 shuts it at once.
enum { GATE_UNDECIDED = 0, GATE_OPEN = 1, GATE_SHUT = 2 };
__device__ __forceinline__ bool grid_gate(CGState *st, int limit, const HostPost &post,
                                          int *ok_sh) {
  __syncthreads();
  if (threadIdx.x == 0) {
    bool shut = limit <= 0 && atomicCAS(&st->gate, GATE_UNDECIDED, GATE_SHUT) == GATE_UNDECIDED;
    __threadfence();
    if (atomicAdd(&st->gbar, 1u) + 1u == gridDim.x) {
      __threadfence();
      atomicCAS(&st->gate, GATE_UNDECIDED, GATE_OPEN);
    }
    int g = GATE_UNDECIDED;
    for (int n = 0; n < limit && g == GATE_UNDECIDED; ++n)
      asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(g) : "l"(&st->gate) : "memory");
    if (g == GATE_UNDECIDED) {
      g = atomicCAS(&st->gate, GATE_UNDECIDED, GATE_SHUT);
      if (g == GATE_UNDECIDED) {
        g = GATE_SHUT;
        shut = true;
      }
      __threadfence();
    }
    if (shut) {
      post.hr->done = CG_LEFT;
      __threadfence_system();
      *(volatile unsigned int *)&post.hr->cg_seq = post.seq;
    }
    *ok_sh = g == GATE_OPEN;
  }
  __syncthreads();
  return *ok_sh != 0;
}

__device__ __forceinline__ void post_outcome(const HostPost &post, const CGState *st) {
  HostResult *h = post.hr;
  h->done = st->done;
  h->iters = st->iters;
  h->resMax = st->resMax;
  h->retResidual = st->retResidual;
  h->resIni = st->resIni;
  __threadfence_system();
  *(volatile unsigned int *)&h->cg_seq = post.seq;
}

// NTH threads; M groups per block, K cells of a group per thread at most when
// QREG (A p in registers, otherwise in qg); GS: the gradient is kept in shared
// memory too.  GV groups in all.
template <int NTH, int M, int K, bool QREG, bool GS, class GT>
__global__ void __launch_bounds__(NTH, 1)
k_cg_resident(float4 *x, const float4 *__restrict__ r0, float4 *p, float4 *qg,
              const GT *__restrict__ g, Dims4 d, BoxDecoder bx, uint32_t nint, uint32_t per,
              int GV, OFConsts c, CGState *st, double *part, int maxIter, int polls, int *err,
              HostPost post) {
  extern __shared__ float4 res_sm[];
  __shared__ FF shff[3][NTH / 32];
  __shared__ float shm[NTH / 32];
  __shared__ double fin[5];
  __shared__ float ab[2];
  __shared__ int ok, stop;
  if (st->done != CG_RUNNING) {  // the same for every block
    if (blockIdx.x == 0 && threadIdx.x == 0) post_outcome(post, st);
    return;
  }
  // the block's cells are contiguous; group v of it covers per cells from
  // first(v)
  const uint32_t b0 = blockIdx.x * (M * per);
  auto first = [&](int v) { return min(b0 + v * per, nint); };
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float4 *rs = res_sm, *gsm = res_sm + M * per;
  const idx_t sY = d.x, sZ = d.sz(), sT = d.st();
  double *pA = part, *pB = part + 3 * GV;  // [dot][group]; [parity][z.r, max r][group]
  const double acc = st->acc, sigma0 = st->sigma;
  auto addr = [&](uint32_t n) {
    int i, j, k, l;
    bx.decode(n, i, j, k, l);
    return d.index(i, j, k, l);
  };
  int ids[QREG ? M * K : 1];
  float4 q[QREG ? M * K : 1];
#pragma unroll
  for (int v = 0; v < M; ++v) {
    const uint32_t c0 = first(v), c1 = first(v + 1);
    for (uint32_t n = c0 + threadIdx.x; n < c1; n += NTH) {
      const idx_t id = addr(n);
      rs[n - b0] = __ldg(r0 + id);
      if (GS) gsm[n - b0] = ld_g(g, id);
    }
    if (QREG) {
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const uint32_t n = c0 + threadIdx.x + k * NTH;
        ids[v * K + k] = n < c1 ? (int)addr(n) : 0;
      }
    }
  }
  // (each thread reads back only the shared cells that it wrote)

  unsigned int target = 0;
  for (int it = 0;; ++it) {
    FF d0, d1, d2;
    auto phase1 = [&](uint32_t n, idx_t id) {
      const float4 pc = p[id];
      const float4 tm = p[id - sT], zm = p[id - sZ], ym = p[id - sY], xm = p[id - 1];
      const float4 xp = p[id + 1], yp = p[id + sY], zp = p[id + sZ], tp = p[id + sT];
      const float4 gg = GS ? gsm[n - b0] : ld_g(g, id);
      const float4 r = rs[n - b0];
      const float gp = __fmaf_rn(gg.w, pc.w, __fmaf_rn(gg.z, pc.z, __fmaf_rn(gg.y, pc.y, gg.x * pc.x)));
      auto row = [&](float gc, float p0, float a0, float a1, float a2, float a3, float a4, float a5,
                     float a6, float a7) {
        const float nb = ((a0 + a1) + (a2 + a3)) + ((a4 + a5) + (a6 + a7));
        return __fmaf_rn(gp, gc, __fmaf_rn(c.offd, nb, c.diag * p0));
      };
      float4 qq;
      qq.x = row(gg.x, pc.x, tm.x, zm.x, ym.x, xm.x, xp.x, yp.x, zp.x, tp.x);
      qq.y = row(gg.y, pc.y, tm.y, zm.y, ym.y, xm.y, xp.y, yp.y, zp.y, tp.y);
      qq.z = row(gg.z, pc.z, tm.z, zm.z, ym.z, xm.z, xp.z, yp.z, zp.z, tp.z);
      qq.w = row(gg.w, pc.w, tm.w, zm.w, ym.w, xm.w, xp.w, yp.w, zp.w, tp.w);
      const float4 pre = make_float4(rcp_newton(gg.x * gg.x + c.diag), rcp_newton(gg.y * gg.y + c.diag),
                                     rcp_newton(gg.z * gg.z + c.diag), rcp_newton(gg.w * gg.w + c.diag));
      ff_add(d0, pc.x * qq.x);
      ff_add(d0, pc.y * qq.y);
      ff_add(d0, pc.z * qq.z);
      ff_add(d0, pc.w * qq.w);
      const float ux = pre.x * qq.x, uy = pre.y * qq.y, uz = pre.z * qq.z, uw = pre.w * qq.w;
      ff_add(d1, ux * r.x);
      ff_add(d1, uy * r.y);
      ff_add(d1, uz * r.z);
      ff_add(d1, uw * r.w);
      ff_add(d2, ux * qq.x);
      ff_add(d2, uy * qq.y);
      ff_add(d2, uz * qq.z);
      ff_add(d2, uw * qq.w);
      return qq;
    };
#pragma unroll
    for (int v = 0; v < M; ++v) {
      const uint32_t c0 = first(v), c1 = first(v + 1);
      d0 = d1 = d2 = FF{0.f, 0.f};
      if (QREG) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const uint32_t n = c0 + threadIdx.x + k * NTH;
          if (n < c1) q[v * K + k] = phase1(n, ids[v * K + k]);
        }
      } else {
#pragma unroll 2
        for (uint32_t n = c0 + threadIdx.x; n < c1; n += NTH) {
          const idx_t id = addr(n);
          qg[id] = phase1(n, id);
        }
      }
      d0 = warp_sum_ff(d0);
      d1 = warp_sum_ff(d1);
      d2 = warp_sum_ff(d2);
      if (v > 0) __syncthreads();  // the last group's sums have been read
      if (lane == 0) {
        shff[0][w] = d0;
        shff[1][w] = d1;
        shff[2][w] = d2;
      }
      __syncthreads();
      if (w < 3 && c0 < nint) {
        const FF t = warp_sum_ff(lane < NTH / 32 ? shff[w][lane] : FF{0.f, 0.f});
        if (lane == 0) __stcg(pA + w * GV + blockIdx.x * M + v, ff_value(t));
      }
    }
    target += gridDim.x;
    if (it == 0) {  // nothing but q and part has been written
      if (!grid_gate(st, polls, post, &ok)) return;
    } else if (!grid_barrier(&st->gbar, target, &ok)) {
      if (threadIdx.x == 0) *(volatile int *)err = FLOF_DEV_ERR_GRID_TIMEOUT;
      return;
    }
    // the sums over the groups: p.q, q.z, q.M^-1 q of this iteration, z.r and
    // max r of the iterate that the last phase 2 left
    const int par = it & 1;
    if (w < 5) {
      const double *src = w < 3 ? pA + w * GV : pB + (2 * par + (w - 3)) * GV;
      double s = 0.0;
      if (w < 4) {
        if (w < 3 || it > 0)
          for (int b = lane; b < GV; b += 32) s += __ldcg(src + b);
        s = warp_sum(s);
      } else {
        float m = 0.f;  // border rows hold r = 0
        if (it > 0)
          for (int b = lane; b < GV; b += 32) m = fmaxf(m, (float)__ldcg(src + b));
        s = (double)warp_max(m);
      }
      if (lane == 0) fin[w] = s;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      int sp = 0;
      if (it > 0 && fin[4] <= acc) sp = CG_CONVERGED;
      else if (it >= maxIter) sp = CG_MAXITER;
      stop = sp;
      if (!sp) {
        const double sg = it > 0 ? fin[3] : sigma0;
        const float af = quotient(sg, fin[0]);
        const double a = (double)af;
        ab[0] = af;
        const double zr = fma(a * a, fin[2], fma(-2.0 * a, fin[1], sg));
        ab[1] = zr < CG_BETA_FLOOR * sg ? 0.f : quotient(zr, sg);
      }
    }
    __syncthreads();
    if (stop) {
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        st->done = stop;
        st->iters = it;
        st->resMax = (float)fin[4];
        st->retResidual = (float)(fin[4] / st->resIni);
        post_outcome(post, st);
      }
      return;
    }
    const float a = ab[0], b = ab[1];
    FF rz;
    float mx;
    auto phase2 = [&](uint32_t n, idx_t id, const float4 qq) {
      float4 r = rs[n - b0];
      const float4 gg = GS ? gsm[n - b0] : ld_g(g, id);
      const float4 pc = p[id];
      float4 xx = x[id], pn;
      const float4 pre = res_precond(gg, c.diag);
      auto one = [&](float &rc, float &xc, float &pc1, float p0, float q0, float m0) {
        rc = __fmaf_rn(-a, q0, rc);
        const float z = rc * m0;
        xc = __fmaf_rn(a, p0, xc);
        pc1 = __fmaf_rn(b, p0, z);
        ff_add(rz, z * rc);
        mx = fmaxf(mx, rc);
      };
      one(r.x, xx.x, pn.x, pc.x, qq.x, pre.x);
      one(r.y, xx.y, pn.y, pc.y, qq.y, pre.y);
      one(r.z, xx.z, pn.z, pc.z, qq.z, pre.z);
      one(r.w, xx.w, pn.w, pc.w, qq.w, pre.w);
      rs[n - b0] = r;
      x[id] = xx;
      p[id] = pn;
    };
#pragma unroll
    for (int v = 0; v < M; ++v) {
      const uint32_t c0 = first(v), c1 = first(v + 1);
      rz = FF{0.f, 0.f};
      mx = 0.f;
      if (QREG) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const uint32_t n = c0 + threadIdx.x + k * NTH;
          if (n < c1) phase2(n, ids[v * K + k], q[v * K + k]);
        }
      } else {
#pragma unroll 2
        for (uint32_t n = c0 + threadIdx.x; n < c1; n += NTH) {
          const idx_t id = addr(n);
          phase2(n, id, qg[id]);
        }
      }
      rz = warp_sum_ff(rz);
      mx = warp_max(mx);
      if (v > 0) __syncthreads();
      if (lane == 0) {
        shff[0][w] = rz;
        shm[w] = mx;
      }
      __syncthreads();
      if (c0 < nint) {
        if (w == 0) {
          const FF t = warp_sum_ff(lane < NTH / 32 ? shff[0][lane] : FF{0.f, 0.f});
          if (lane == 0) __stcg(pB + 2 * (par ^ 1) * GV + blockIdx.x * M + v, ff_value(t));
        } else if (w == 1) {
          const float t = warp_max(lane < NTH / 32 ? shm[lane] : 0.f);
          if (lane == 0) __stcg(pB + (2 * (par ^ 1) + 1) * GV + blockIdx.x * M + v, (double)t);
        }
      }
    }
    target += gridDim.x;
    if (!grid_barrier(&st->gbar, target, &ok)) {
      if (threadIdx.x == 0) *(volatile int *)err = FLOF_DEV_ERR_GRID_TIMEOUT;
      return;
    }
  }
}

struct ResidentArgs {
  float4 *x, *r, *p, *q;
  Dims4 d;
  uint32_t n, per;  // interior cells, cells per group
  OFConsts c;
  CGState *st;
  double *part;
  int maxIter, polls;
  int *err;
  HostPost post;
  cudaStream_t s;
};

template <int NTH, int M, int K, bool QREG, bool GS, class GT>
bool launch_one(ResidentArgs a, const GT *g, ResidentShare &share) {
  auto k = k_cg_resident<NTH, M, K, QREG, GS, GT>;
  constexpr size_t per_cell = GS ? 32 : 16;
  // the shared memory that the kernel may use, asked for once per device; 0
  // when the device refuses it
  static PerDevice<size_t> asked;
  const size_t smem_max = asked.get(current_device(), [&]() -> size_t {
    int n = 0;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, RESIDENT_SMEM) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, NTH, RESIDENT_SMEM) != cudaSuccess ||
        n < 1) {
      cudaGetLastError();
      return 0;
    }
    return RESIDENT_SMEM;
  });
  const size_t smem = per_cell * a.per * M;
  if (smem > smem_max) return false;
  BoxDecoder bx = make_decoder(a.d.x - 2, a.d.y - 2, a.d.z - 2, 1, 1, 1, 1);
  const float4 *r0 = a.r;
  int groups = (int)((a.n + a.per - 1) / a.per);
  const int grid = (groups + M - 1) / M;
  void *args[] = {&a.x, &r0,  &a.p, &a.q,  &g,    &a.d,       &bx,    &a.n,   &a.per,
                  &groups, &a.c, &a.st, &a.part, &a.maxIter, &a.polls, &a.err, &a.post};
  share.take(grid);
  if (cudaLaunchCooperativeKernel((const void *)k, dim3(grid), dim3(NTH), args, smem, a.s) !=
      cudaSuccess) {
    cudaGetLastError();
    share.give();
    return false;
  }
  return true;
}

template <class GT>
bool launch_any(ResidentArgs a, const GT *g, bool shared, ResidentShare &share) {
  if (!resident_cells_ok(a.d) || a.maxIter <= 0) return false;
  a.n = (uint32_t)((long long)(a.d.x - 2) * (a.d.y - 2) * (a.d.z - 2) * (a.d.t - 2));
  const uint32_t sms = (uint32_t)sm_count();
  // 256 cells per group until every SM has one (fewer groups make the barriers
  // and the sums over them cheaper: 6.2 against 6.9 us for 6000 cells), then
  // two cells for each of 512 threads, then up to six for each of 1024, then
  // A p and the gradient out of registers and shared memory.  The larger
  // levels fill the SMs alone and are not shared out.
  a.per = (a.n + sms - 1) / sms;
  if (a.per <= 256) {
    a.per = 256;
    return shared ? launch_one<256, 4, 1, true, true>(a, g, share)
                  : launch_one<256, 1, 1, true, true>(a, g, share);
  }
  if (a.per <= 1024)
    return shared ? launch_one<512, 4, 2, true, true>(a, g, share)
                  : launch_one<512, 1, 2, true, true>(a, g, share);
  if (a.per <= 6144) return launch_one<1024, 1, 6, true, true>(a, g, share);
  return launch_one<1024, 1, 1, false, false>(a, g, share);
}

}  // namespace

bool resident_cells_ok(Dims4 d) {
  if (d.x < 3 || d.y < 3 || d.z < 3 || d.t < 3) return false;
  const long long n = (long long)(d.x - 2) * (d.y - 2) * (d.z - 2) * (d.t - 2);
  return n <= (long long)sm_count() * (long long)(RESIDENT_SMEM / 16);
}

void ResidentShare::take(int n) {
  shares = &sm_shares(current_device());
  shares->acquire(n, sm_count());
  blocks = n;
}
void ResidentShare::give() {
  if (blocks) shares->release(blocks);
  blocks = 0;
}

bool launch_cg_resident(float4 *x, float4 *r, float4 *p, float4 *q, const float4 *g, Dims4 d,
                        OFConsts c, CGState *st, double *part, int maxIter, int polls, int *err,
                        HostPost post, bool shared, ResidentShare &share, cudaStream_t s) {
  return launch_any(ResidentArgs{x, r, p, q, d, 0, 0, c, st, part, maxIter, polls, err, post, s}, g,
                    shared, share);
}
bool launch_cg_resident(float4 *x, float4 *r, float4 *p, float4 *q, const BF4 *g, Dims4 d,
                        OFConsts c, CGState *st, double *part, int maxIter, int polls, int *err,
                        HostPost post, bool shared, ResidentShare &share, cudaStream_t s) {
  return launch_any(ResidentArgs{x, r, p, q, d, 0, 0, c, st, part, maxIter, polls, err, post, s}, g,
                    shared, share);
}

}  // namespace flof
