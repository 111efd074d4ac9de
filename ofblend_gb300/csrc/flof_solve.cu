// flof_solve.cu -- optical-flow system assembly, Jacobi-PCG, Gaussian velocity
// blur and the level-set projection correction.
//
// Reference: source/plugin/optflow4d.cpp
//   opticalFlowDim        :361-553   (assembly :398-493, copy back :520-529)
//   FixedMatrixOF/applyMat :179-232  (matrix-free here: the block is g g^T +
//                                     diag I, rebuilt from the stored g)
//   GridCGOptflow4d        :268-355
//   knGaussianBlur         :132-158
//   knProjectCells et al.  :651-734
//   knCvExpolBlur4d        :613-626
#include <float.h>

#include <algorithm>

#include "flof_kernels.h"

namespace flof {

constexpr int NT = 256;

// ---------------------------------------------------------------------------
// Assembly + PCG initialisation
// ---------------------------------------------------------------------------

static inline BoxDecoder interior_decoder(Dims4 d) {
  return make_decoder(d.x - 2 > 0 ? d.x - 2 : 1, d.y - 2 > 0 ? d.y - 2 : 1,
                      d.z - 2 > 0 ? d.z - 2 : 1, 1, 1, 1, 1);
}
static inline uint32_t interior_count(Dims4 d) {
  if (d.x < 3 || d.y < 3 || d.z < 3 || d.t < 3) return 0;
  return (uint32_t)((long long)(d.x - 2) * (d.y - 2) * (d.z - 2) * (d.t - 2));
}

// Jacobi preconditioner of row (cell,d): 1/blockd[d][d] with the diagonal
// g_d*g_d + diag, rounded like the reference's (float)(1./diag).
__device__ __forceinline__ float4 precond_of(const float4 g, float diag) {
  float4 p;
  p.x = __frcp_rn(g.x * g.x + diag);
  p.y = __frcp_rn(g.y * g.y + diag);
  p.z = __frcp_rn(g.z * g.z + diag);
  p.w = __frcp_rn(g.w * g.w + diag);
  return p;
}

__global__ void __launch_bounds__(NT)
k_of_assemble_init(const float *__restrict__ i0w, const float *__restrict__ i1,
                   const float4 *__restrict__ vel, float4 *__restrict__ g,
                   float4 *__restrict__ r, float4 *__restrict__ p,
                   float4 *__restrict__ x, Dims4 d, BoxDecoder bx, uint32_t ncells,
                   OFConsts c, float accuracy, CGState *st, double *dpart,
                   float *fpart) {
  __shared__ double shd[NT / 32];
  __shared__ FF shff[NT / 32];
  __shared__ float shf[NT / 32];
  FF dot = {0.f, 0.f};
  float mx = -FLT_MAX;
  const idx_t sY = d.x, sZ = d.sz(), sT = d.st();
  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < ncells;
       q += gridDim.x * blockDim.x) {
    int i, j, k, l;
    bx.decode(q, i, j, k, l);
    const idx_t id = q;
    x[id] = zero4;  // setConst(result, 0) (optflow4d.cpp:280)
    if (!in_bounds(d, i, j, k, l, 1)) {
      // identity rows with zero rhs (optflow4d.cpp:424-433): g = r = p = 0
      g[id] = zero4;
      r[id] = zero4;
      p[id] = zero4;
      continue;
    }
    const float tderiv = (__ldg(i1 + id) - __ldg(i0w + id)) / c.mDt;
    float gr[4];
    gr[0] = (__ldg(i1 + id + 1) - __ldg(i1 + id - 1)) * c.dxf;
    gr[1] = (__ldg(i1 + id + sY) - __ldg(i1 + id - sY)) * c.dxf;
    gr[2] = (__ldg(i1 + id + sZ) - __ldg(i1 + id - sZ)) * c.dxf;
    gr[3] = (__ldg(i1 + id + sT) - __ldg(i1 + id - sT)) * c.dxf;
    float rh[4];
#pragma unroll
    for (int dd = 0; dd < 4; ++dd) rh[dd] = -gr[dd] * tderiv;
    if (vel) {
      // rhs -= wSmooth (v - v_nb) mDx mDx2Inv for m = -t,-z,-y,-x,+x,+y,+z,+t,
      // then -= wEnergy v mDx (optflow4d.cpp:450-478)
      const float4 vc = __ldg(vel + id);
      const idx_t off[8] = {-sT, -sZ, -sY, -1, 1, sY, sZ, sT};
      const float vcc[4] = {vc.x, vc.y, vc.z, vc.w};
#pragma unroll
      for (int m = 0; m < 8; ++m) {
        const float4 vn = __ldg(vel + id + off[m]);
        const float vnn[4] = {vn.x, vn.y, vn.z, vn.w};
#pragma unroll
        for (int dd = 0; dd < 4; ++dd)
          rh[dd] -= c.wSmooth * (vcc[dd] - vnn[dd]) * c.mDx * 1.0f;
      }
#pragma unroll
      for (int dd = 0; dd < 4; ++dd) rh[dd] -= c.wEnergy * vcc[dd] * c.mDx;
    }
    const float4 gg = make_float4(gr[0], gr[1], gr[2], gr[3]);
    const float4 rr = make_float4(rh[0], rh[1], rh[2], rh[3]);
    const float4 pre = precond_of(gg, c.diag);
    const float4 z = make_float4(rr.x * pre.x, rr.y * pre.y, rr.z * pre.z, rr.w * pre.w);
    g[id] = gg;
    r[id] = rr;
    p[id] = z;
    ff_add(dot, z.x * rr.x);
    ff_add(dot, z.y * rr.y);
    ff_add(dot, z.z * rr.z);
    ff_add(dot, z.w * rr.w);
    mx = fmaxf(mx, fmaxf(fmaxf(rr.x, rr.y), fmaxf(rr.z, rr.w)));
  }
  const double bd = block_sum_ff<NT>(dot, shff);
  const float bm = block_max<NT>(mx, shf);
  if (threadIdx.x == 0) {
    dpart[blockIdx.x] = bd;
    fpart[blockIdx.x] = bm;
  }
  if (last_block_arrives(&st->counter[0])) {
    double s = 0.0;
    float m = 0.0f;  // border rows hold r = 0
    for (int q = threadIdx.x; q < (int)gridDim.x; q += blockDim.x) {
      s += __ldcg(dpart + q);
      m = fmaxf(m, __ldcg(fpart + q));
    }
    s = block_sum<NT>(s, shd);
    m = block_max<NT>(m, shf);
    if (threadIdx.x == 0) {
      const double residual = (double)m;
      st->resIni = residual;
      st->resMax = m;
      st->iters = 0;
      st->gbar = 0;
      st->gate = 0;
      st->counter[0] = 0;
      if (residual < (double)1e-6f) {
        st->retResidual = 0.f;
        st->done = CG_EARLY;
      } else {
        st->acc = (double)accuracy * residual;
        st->sigma = s;
        if (s == 0.0 || s != s) {
          st->retResidual = 1e10f;  // the caller's initial cgRes stays
          st->done = CG_FAILED_SIGMA;
        } else {
          st->retResidual = 1.0f;   // residual / resIni before any iteration
          st->done = CG_RUNNING;
        }
      }
    }
  }
}

void launch_of_assemble_init(const float *i0w, const float *i1,
                             const float4 *vel, float4 *g, float4 *r,
                             float4 *p, float4 *x, Dims4 d, OFConsts c,
                             float accuracy, CGState *st, double *dpart,
                             float *fpart, cudaStream_t s) {
  // five blocks per SM are resident: a single wave (mean over the levels of a
  // 64^4 solve 82 us; 8 per SM 95, 10 per SM 90, one trip per thread 172)
  k_of_assemble_init<<<grid_for(d.cells(), NT, 5), NT, 0, s>>>(
      i0w, i1, vel, g, r, p, x, d, make_decoder(d.x, d.y, d.z, 0, 0, 0, 0),
      (uint32_t)d.cells(), c, accuracy, st, dpart, fpart);
}

// ---------------------------------------------------------------------------
// PCG iteration (GridCGOptflow4d::solve, optflow4d.cpp:304-326)
// ---------------------------------------------------------------------------

// q = A p over the interior rows; applyMat order: 8 neighbour terms
// (-t,-z,-y,-x,+x,+y,+z,+t) then the 4 block terms.
//
// A thread owns one interior (x,y) column cell at one z and walks MV_TT
// consecutive t planes, keeping p at t-1, t and t+1 in registers, so the -t
// and +t terms cost no extra load, and loading the next plane's operands
// while it computes the current one.  A work item is (run of MV_RUN cells of
// the interior (x,y) plane, MV_ZB planes z, t chunk) with the (x,y) run
// fastest, so the blocks resident at one time cover neighbouring z at the same
// t chunk and the z-neighbour loads hit L2.  The grid is persistent (a fixed number of
// blocks per SM); p.Ap is accumulated per thread in float-float and summed
// in double by the last block to finish, in a fixed order.
//
// MV_DOTS (the plain PCG): the kernel also forms q.M^-1 q, from which its last
// block predicts the next z.r, and so beta, before r is updated (cg_scalars).
// The step kernel then has alpha and beta and updates r and p in one pass.
// The extra sum costs 8 us of 144 at 64^4.  The loads need the 1024 threads per
// SM that 64 registers allow: at 105 registers it takes 186 us.  Two z planes a
// block share their z neighbours in L1 (148 -> 146 us at 64^4, 59 -> 57 at 48^4; four planes 150 and 61, rows of
// 256 cells 152 and 59), the fused rows take 146 -> 142 and 57 -> 56 and halve
// the rounding (the 64^4 deformation against 64 bits 7.5e-7 -> 4.8e-7).  Each
// product of q.M^-1 q enters the float-float sum by itself, like those of every
// other dot product, with a reciprocal that has no common error (rcp_newton):
// 142 -> 144 us.
constexpr int MV_RUN = 128;
constexpr int MV_ZB = 2;
constexpr int MV_NT = MV_RUN * MV_ZB;
// What a matvec computes: the reference's operations in its order and p.q
// (strict mode, whose rows are applyMat's bit for bit), the same rows with
// fused operations, or those and q.M^-1 q.
enum { MV_REFERENCE = 0, MV_FUSED = 1, MV_DOTS = 2 };

// alpha, and beta before the step that it belongs to.  With r' = r - a q,
//   z'.r' = z.r - 2 a q.z + a^2 q.M^-1 q,
// where q.z is not summed but follows from p.q: z = p - b p_old (b and p_old
// the last step's), so q.z = p.q - b q.p_old.  q.p_old is zero but for
// rounding; that rounding must not be left out, as each step would double it.
// It is known from the last step's sums (A symmetric, q_old = (r_old - r) / a_old,
// and the sigma that the step summed afresh from the updated r):
//   q.p_old = p.q_old = z.q_old + b p_old.q_old,
//   z.q_old = (z.r_old - z.r) / a_old,  z.r_old = z_old.r = z_old.r_old - a_old q_old.z_old.
// So no error passes from one beta to the next but the rounding of the vectors.
// alpha itself uses the fresh sigma.
// The terms are of the size of z.r, whatever is left of it, so beta's error is
// that of the sums: 2^-24 (1 + beta) over the root of their number of products
// (1e-9 measured from 0.01M cells on), below beta's own rounding to float
// unless a single step takes more than nine tenths of z.r away.  A beta below
// CG_BETA_FLOOR is noise, which the next one's q.p_old would carry on: the
// iteration starts anew from p = z.
__device__ __forceinline__ void cg_scalars(CGState *st, double pq, double qmq, int slot) {
  const double sg = st->sigma;
  st->pAp = pq;
  st->alpha = sg / pq;
  st->alphaf = (float)st->alpha;
  st->al[slot] = st->alphaf;
  const double a = (double)st->alphaf;  // the value the step uses
  double qz = pq;
  if (st->iters > 0) {
    const double ao = st->aOld, bo = (double)st->betaf;
    const double zro = st->sgOld - ao * st->qzOld;
    qz -= bo * ((zro - sg) / ao + bo * st->pqOld);
  }
  const double b = fma(a * a, qmq, fma(-2.0 * a, qz, sg)) / sg;
  st->beta = b < CG_BETA_FLOOR ? 0.0 : b;  // a NaN stays
  st->betaf = (float)st->beta;
  st->aOld = a;
  st->sgOld = sg;
  st->qzOld = qz;
  st->pqOld = pq;
}

struct MVShape {
  FastDiv fx;        // interior x extent
  int nxy;           // interior (x,y) cells
  int runs;          // ceil(nxy / MV_RUN)
  FastDiv fruns, fz;  // runs, groups of MV_ZB interior z planes
  int items;         // runs * z groups * tchunks
};

__device__ __forceinline__ void mv_acc(float4 &v, float o, const float4 a) {
  v.x += o * a.x;
  v.y += o * a.y;
  v.z += o * a.z;
  v.w += o * a.w;
}

// The operands of one cell other than p at t-1 and t.
struct MVLoads {
  float4 pp, gg, zm, ym, xm, xp, yp, zp;
};
template <class GT>
__device__ __forceinline__ void mv_load(MVLoads &a, const float4 *__restrict__ p,
                                        const GT *__restrict__ g, idx_t id, idx_t sY,
                                        idx_t sZ, idx_t sT) {
  a.pp = __ldg(p + id + sT);
  a.gg = ld_g(g, id);
  a.zm = __ldg(p + id - sZ);
  a.ym = __ldg(p + id - sY);
  a.xm = __ldg(p + id - 1);
  a.xp = __ldg(p + id + 1);
  a.yp = __ldg(p + id + sY);
  a.zp = __ldg(p + id + sZ);
}

// OFFD: the neighbour terms are present (applyMat skips them for a zero
// off-diagonal, optflow4d.cpp:215).  MV_TT: t planes per work item.
template <bool OFFD, int MV_TT, int MODE, class GT>
__global__ void __launch_bounds__(MV_NT, 1024 / MV_NT)
k_cg_matvec(const float4 *__restrict__ p, const GT *__restrict__ g,
            float4 *__restrict__ q, Dims4 d, MVShape sh, OFConsts c, CGState *st,
            double *dpart, int slot) {
  pdl_wait();
  pdl_launch_dependents();
  if (st->done) return;
  __shared__ double shd[MV_NT / 32];
  __shared__ FF shff[MV_NT / 32];
  FF dot = {0.f, 0.f}, dotm = {0.f, 0.f};
  const idx_t sY = d.x, sZ = d.sz(), sT = d.st();
  const float o = c.offd;
  for (int item = blockIdx.x; item < sh.items; item += gridDim.x) {
    const uint32_t r1 = sh.fruns.div((uint32_t)item);
    const int run = item - (int)r1 * sh.runs;
    const uint32_t tc = sh.fz.div(r1);
    const int k = 1 + (int)(r1 - tc * sh.fz.d) * MV_ZB + (int)threadIdx.x / MV_RUN;
    const int n = run * MV_RUN + (int)threadIdx.x % MV_RUN;
    if (n >= sh.nxy || k >= d.z - 1) continue;
    const uint32_t jj = sh.fx.div((uint32_t)n);
    const int i = 1 + (n - (int)(jj * sh.fx.d)), j = 1 + (int)jj;
    const int l0 = 1 + (int)tc * MV_TT;
    const int l1 = min(l0 + MV_TT, d.t - 1);
    idx_t id = d.index(i, j, k, l0);
    float4 pm = __ldg(p + id - sT), pc = __ldg(p + id);
    MVLoads cur, nxt;
    mv_load(cur, p, g, id, sY, sZ, sT);
    for (int l = l0; l < l1; ++l, id += sT) {
      // the last plane reloads its own operands instead of reading past l1
      mv_load(nxt, p, g, l + 1 < l1 ? id + sT : id, sY, sZ, sT);
      float4 qq;
      if (MODE == MV_REFERENCE) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (OFFD) {
          mv_acc(v, o, pm);
          mv_acc(v, o, cur.zm);
          mv_acc(v, o, cur.ym);
          mv_acc(v, o, cur.xm);
          mv_acc(v, o, cur.xp);
          mv_acc(v, o, cur.yp);
          mv_acc(v, o, cur.zp);
          mv_acc(v, o, cur.pp);
        }
        const float gv[4] = {cur.gg.x, cur.gg.y, cur.gg.z, cur.gg.w};
        const float pv[4] = {pc.x, pc.y, pc.z, pc.w};
        float vv[4] = {v.x, v.y, v.z, v.w};
  #pragma unroll
        for (int dd = 0; dd < 4; ++dd) {
  #pragma unroll
          for (int m = 0; m < 4; ++m) {
            float b = gv[dd] * gv[m];
            if (dd == m) b = b + c.diag;
            vv[dd] += b * pv[m];
          }
        }
        qq = make_float4(vv[0], vv[1], vv[2], vv[3]);
      } else {
        // row c of g g^T + diag I and the neighbours' sum: 45 operations a cell
        // in place of 116
        const float gp = __fmaf_rn(
            cur.gg.w, pc.w, __fmaf_rn(cur.gg.z, pc.z, __fmaf_rn(cur.gg.y, pc.y, cur.gg.x * pc.x)));
        auto row = [&](float gc, float p0, float a0, float a1, float a2, float a3, float a4,
                       float a5, float a6, float a7) {
          float t = c.diag * p0;
          if (OFFD) t = __fmaf_rn(o, ((a0 + a1) + (a2 + a3)) + ((a4 + a5) + (a6 + a7)), t);
          return __fmaf_rn(gp, gc, t);
        };
        qq.x = row(cur.gg.x, pc.x, pm.x, cur.zm.x, cur.ym.x, cur.xm.x, cur.xp.x, cur.yp.x,
                   cur.zp.x, cur.pp.x);
        qq.y = row(cur.gg.y, pc.y, pm.y, cur.zm.y, cur.ym.y, cur.xm.y, cur.xp.y, cur.yp.y,
                   cur.zp.y, cur.pp.y);
        qq.z = row(cur.gg.z, pc.z, pm.z, cur.zm.z, cur.ym.z, cur.xm.z, cur.xp.z, cur.yp.z,
                   cur.zp.z, cur.pp.z);
        qq.w = row(cur.gg.w, pc.w, pm.w, cur.zm.w, cur.ym.w, cur.xm.w, cur.xp.w, cur.yp.w,
                   cur.zp.w, cur.pp.w);
      }
      q[id] = qq;
      ff_add(dot, pc.x * qq.x);
      ff_add(dot, pc.y * qq.y);
      ff_add(dot, pc.z * qq.z);
      ff_add(dot, pc.w * qq.w);
      if (MODE == MV_DOTS) {
        ff_add(dotm, (rcp_newton(cur.gg.x * cur.gg.x + c.diag) * qq.x) * qq.x);
        ff_add(dotm, (rcp_newton(cur.gg.y * cur.gg.y + c.diag) * qq.y) * qq.y);
        ff_add(dotm, (rcp_newton(cur.gg.z * cur.gg.z + c.diag) * qq.z) * qq.z);
        ff_add(dotm, (rcp_newton(cur.gg.w * cur.gg.w + c.diag) * qq.w) * qq.w);
      }
      pm = pc;
      pc = cur.pp;
      cur = nxt;
    }
  }
  const double bd = block_sum_ff<MV_NT>(dot, shff);
  const double bm = MODE == MV_DOTS ? block_sum_ff<MV_NT>(dotm, shff) : 0.0;
  if (threadIdx.x == 0) {
    dpart[blockIdx.x] = bd;
    if (MODE == MV_DOTS) dpart[gridDim.x + blockIdx.x] = bm;
  }
  if (last_block_arrives(&st->counter[1])) {
    double s = 0.0, sm = 0.0;
    for (int q2 = threadIdx.x; q2 < (int)gridDim.x; q2 += blockDim.x) {
      s += __ldcg(dpart + q2);
      if (MODE == MV_DOTS) sm += __ldcg(dpart + gridDim.x + q2);
    }
    s = block_sum<MV_NT>(s, shd);
    if (MODE == MV_DOTS) sm = block_sum<MV_NT>(sm, shd);
    if (threadIdx.x == 0) {
      if (MODE == MV_DOTS) {
        cg_scalars(st, s, sm, slot);
      } else {
        st->pAp = s;
        st->alpha = st->sigma / s;
        st->alphaf = (float)st->alpha;
      }
      st->counter[1] = 0;
    }
  }
}

namespace {

template <bool OFFD, int TT, int MODE, class GT>
void matvec_variant(const float4 *p, const GT *g, float4 *q, Dims4 d, OFConsts c,
                    CGState *st, double *dpart, cudaStream_t s, int slot) {
  MVShape sh;
  const int ex = d.x > 2 ? d.x - 2 : 1, ey = d.y > 2 ? d.y - 2 : 1;
  const int ez = d.z > 2 ? d.z - 2 : 1;
  const int tchunks = d.t > 2 ? (d.t - 2 + TT - 1) / TT : 0;
  const bool empty = d.x < 3 || d.y < 3 || d.z < 3 || d.t < 3;
  sh.fx = FastDiv((uint32_t)ex);
  sh.nxy = empty ? 0 : ex * ey;
  const int zb = (ez + MV_ZB - 1) / MV_ZB;
  sh.runs = (ex * ey + MV_RUN - 1) / MV_RUN;
  sh.fruns = FastDiv((uint32_t)sh.runs);
  sh.fz = FastDiv((uint32_t)zb);
  sh.items = empty ? 0 : sh.runs * zb * tchunks;
  // resident blocks per SM of this instantiation (computed once, thread-safe)
  static const int per_sm = [] {
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_cg_matvec<OFFD, TT, MODE, GT>, MV_NT, 0);
    return n < 1 ? 1 : n;
  }();
  int blocks = sm_count() * per_sm;
  if (blocks > sh.items) blocks = sh.items > 0 ? sh.items : 1;
  launch_pdl(k_cg_matvec<OFFD, TT, MODE, GT>, blocks, MV_NT, s, p, g, q, d, sh, c, st, dpart,
             slot);
}

template <bool OFFD, int MODE, class GT>
void matvec_tt(const float4 *p, const GT *g, float4 *q, Dims4 d, OFConsts c, CGState *st,
               double *dpart, cudaStream_t s, int tt, int slot) {
  if (tt <= 4)
    matvec_variant<OFFD, 4, MODE>(p, g, q, d, c, st, dpart, s, slot);
  else if (tt >= 16)
    matvec_variant<OFFD, 16, MODE>(p, g, q, d, c, st, dpart, s, slot);
  else
    matvec_variant<OFFD, 8, MODE>(p, g, q, d, c, st, dpart, s, slot);
}

template <int MODE, class GT>
void matvec_any(const float4 *p, const GT *g, float4 *q, Dims4 d, OFConsts c, CGState *st,
                double *dpart, cudaStream_t s, const CGTune &tu, int slot) {
  if (c.offd != 0.f)
    matvec_tt<true, MODE>(p, g, q, d, c, st, dpart, s, tu.mv_tt, slot);
  else
    matvec_tt<false, MODE>(p, g, q, d, c, st, dpart, s, tu.mv_tt, slot);
}

}  // namespace

void launch_matvec(const float4 *p, const float4 *g, float4 *q, Dims4 d, OFConsts c, CGState *st,
                   double *dpart, cudaStream_t s, const CGTune &tu) {
  matvec_any<MV_FUSED>(p, g, q, d, c, st, dpart, s, tu, 0);
}
void launch_strict_matvec(const float4 *p, const float4 *g, float4 *q, Dims4 d, OFConsts c,
                          CGState *st, double *dpart, cudaStream_t s) {
  matvec_any<MV_REFERENCE>(p, g, q, d, c, st, dpart, s, CGTune(), 0);
}
void launch_cg_matvec(const float4 *p, const float4 *g, float4 *q, Dims4 d, OFConsts c,
                      CGState *st, double *dpart, int slot, cudaStream_t s, const CGTune &tu) {
  matvec_any<MV_DOTS>(p, g, q, d, c, st, dpart, s, tu, slot);
}
void launch_cg_matvec(const float4 *p, const BF4 *g, float4 *q, Dims4 d, OFConsts c, CGState *st,
                      double *dpart, int slot, cudaStream_t s, const CGTune &tu) {
  matvec_any<MV_DOTS>(p, g, q, d, c, st, dpart, s, tu, slot);
}

// Where the step kernel takes the image gradient g for the Jacobi
// preconditioner from: the stored g (FP32 or BF16), or g rebuilt from
// the target level set i1 with the assembly's own operations (central
// differences times 1/(2 mDx), the same values bit for bit).  i1 is 4 bytes
// per cell against 16 for g; its neighbour loads hit L1 and L2.
template <class T>
struct GradStored {
  const T *__restrict__ g;
  __device__ __forceinline__ float4 operator()(idx_t id) const { return ld_g(g, id); }
};

// r -= alpha q; z = M^-1 r; the next p = z + beta p; sigma' = z.r; max(r); and
// in every CG_RING-th step x += the sum of the last CG_RING alpha p, formed from
// the newest to the oldest.
//
// Bound by HBM: q, r and p read, r and p written, i1 for g (84 bytes a cell),
// and x.  Adding to x in every step reads and writes it each time (32 bytes);
// the directions are kept in CG_RING buffers instead, so that a step in
// CG_RING reads the earlier ones again and x once: (32 + 16 (CG_RING - 1)) /
// CG_RING bytes a step, 20 for four buffers.  The ring's alpha p are added to
// one another before they are added to x, so x is rounded once in four steps
// (with the reference's row operations the 64^4 deformation against 64 bits
// is 7.5e-7 off, 7.9e-7 when every step adds to x).
// An iteration (matvec and step) moves 152 bytes a cell; three kernels (matvec,
// r, then x and p) moved 184.  Step at 64^4: 247 us (6.2 TB/s) with four
// buffers, 259 with two, 270 with one; r and then x and p took 130 + 190 us.
// Iteration: 64^4 463 -> 395 us, 48^4 166 -> 140, 40 x 42 x 38 x 48 107 -> 93.
// The step walks from the last cell to the first: it begins where the matvec
// ended and ends where the next one begins, on q, p and r that L2 still holds
// (64^4 389 -> 386 us an iteration, 48^4 138 -> 135, 40 x 42 x 38 x 48 92 -> 89).
// Keeping x, g or q out of L2 (ld.cs) was slower: 10-20% of the kernel.
// NX: the directions that this step adds to x.  Where memory for a ring is
// short there is one buffer, pin = pout, and every step adds its own (NX = 1);
// a cell is read before it is written, by the same thread.
// FILL: pout is used for the first time in this solve, and the step zeroes its
// border rows too (an eighth of the cells at 64^4, 12 us; clearing the ring's
// three buffers before the first iteration took 120 us, which a solve of one or
// two iterations felt).
__device__ __forceinline__ void axpy4(float4 &x, float a, const float4 p) {
  x.x = __fmaf_rn(a, p.x, x.x);
  x.y = __fmaf_rn(a, p.y, x.y);
  x.z = __fmaf_rn(a, p.z, x.z);
  x.w = __fmaf_rn(a, p.w, x.w);
}

template <int NX, bool FILL, class GS>
__global__ void __launch_bounds__(NT)
k_cg_step(float4 *__restrict__ x, float4 *__restrict__ r, const float4 *__restrict__ q,
          CGRing ring, const float4 *pin, float4 *pout, GS gs, Dims4 d, BoxDecoder bx,
          BoxDecoder rows, uint32_t nint, OFConsts c, CGState *st, double *dpart, float *fpart,
          int maxIter) {
  pdl_wait();
  pdl_launch_dependents();
  if (st->done) return;
  if (FILL) {  // a warp per x row
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const int lane = threadIdx.x & 31;
    const uint32_t n = (uint32_t)d.y * d.z * d.t, warps = gridDim.x * (NT / 32);
    for (uint32_t w = blockIdx.x * (NT / 32) + (threadIdx.x >> 5); w < n; w += warps) {
      int j, k, l, unused;
      rows.decode(w, j, k, l, unused);
      float4 *const row = pout + (idx_t)d.x * w;
      if (j < 1 || j >= d.y - 1 || k < 1 || k >= d.z - 1 || l < 1 || l >= d.t - 1) {
        for (int i = lane; i < d.x; i += 32) row[i] = zero;
      } else if (lane < 2) {
        row[lane ? d.x - 1 : 0] = zero;
      }
    }
  }
  __shared__ double shd[NT / 32];
  __shared__ FF shff[NT / 32];
  __shared__ float shf[NT / 32];
  const float a = st->alphaf, b = st->betaf;
  float al[NX > 1 ? NX : 1];
#pragma unroll
  for (int m = 0; m + 1 < NX; ++m) al[m] = st->al[m];
  FF dot = {0.f, 0.f};
  float mx = -FLT_MAX;
  struct In {
    float4 q, g, r, p, x, po[NX > 1 ? NX - 1 : 1];
  };
  auto load = [&](idx_t id) {
    In v;
    v.q = __ldg(q + id);
    v.r = r[id];
    v.p = pin[id];
    if (NX > 0) {
      v.x = x[id];
#pragma unroll
      for (int m = 0; m + 1 < NX; ++m) v.po[m] = ring.p[m][id];
    }
    v.g = gs(id);
    return v;
  };
  auto cell = [&](idx_t id, const In &v) {
    float4 rr = v.r, pp = v.p;
    axpy4(rr, -a, v.q);
    r[id] = rr;
    const float4 pre = precond_of(v.g, c.diag);
    const float4 z = make_float4(rr.x * pre.x, rr.y * pre.y, rr.z * pre.z, rr.w * pre.w);
    if (NX > 0) {
      float4 t = make_float4(a * pp.x, a * pp.y, a * pp.z, a * pp.w);
#pragma unroll
      for (int m = NX - 2; m >= 0; --m) axpy4(t, al[m], v.po[m]);
      x[id] = make_float4(v.x.x + t.x, v.x.y + t.y, v.x.z + t.z, v.x.w + t.w);
    }
    pp.x = __fmaf_rn(b, pp.x, z.x);
    pp.y = __fmaf_rn(b, pp.y, z.y);
    pp.z = __fmaf_rn(b, pp.z, z.z);
    pp.w = __fmaf_rn(b, pp.w, z.w);
    pout[id] = pp;
    ff_add(dot, z.x * rr.x);
    ff_add(dot, z.y * rr.y);
    ff_add(dot, z.z * rr.z);
    ff_add(dot, z.w * rr.w);
    mx = fmaxf(mx, fmaxf(fmaxf(rr.x, rr.y), fmaxf(rr.z, rr.w)));
  };
  // two cells per trip with all loads issued first, from the last cell down
  const uint32_t stride = gridDim.x * blockDim.x;
  uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
  for (; n + stride < nint; n += 2 * stride) {
    int i, j, k, l;
    bx.decode(nint - 1 - n, i, j, k, l);
    const idx_t i0 = d.index(i, j, k, l);
    bx.decode(nint - 1 - n - stride, i, j, k, l);
    const idx_t i1 = d.index(i, j, k, l);
    const In v0 = load(i0), v1 = load(i1);
    cell(i0, v0);
    cell(i1, v1);
  }
  if (n < nint) {
    int i, j, k, l;
    bx.decode(nint - 1 - n, i, j, k, l);
    const idx_t i0 = d.index(i, j, k, l);
    cell(i0, load(i0));
  }
  const double bd = block_sum_ff<NT>(dot, shff);
  const float bm = block_max<NT>(mx, shf);
  if (threadIdx.x == 0) {
    dpart[blockIdx.x] = bd;
    fpart[blockIdx.x] = bm;
  }
  if (last_block_arrives(&st->counter[2])) {
    double s = 0.0;
    float m = 0.0f;
    for (int q2 = threadIdx.x; q2 < (int)gridDim.x; q2 += blockDim.x) {
      s += __ldcg(dpart + q2);
      m = fmaxf(m, __ldcg(fpart + q2));
    }
    s = block_sum<NT>(s, shd);
    m = block_max<NT>(m, shf);
    if (threadIdx.x == 0) {
      const double residual = (double)m;
      const int iter = st->iters;
      st->resMax = m;
      st->retResidual = (float)(residual / st->resIni);
      st->iters = iter + 1;
      st->counter[2] = 0;
      if (residual <= st->acc) {
        st->done = CG_CONVERGED;
      } else {
        st->sigma = s;
        if (iter + 1 >= maxIter) st->done = CG_MAXITER;
      }
    }
  }
}

// x += the first `count` alpha p of the ring, the ones that no step has added.
__global__ void __launch_bounds__(NT)
k_cg_flush(float4 *__restrict__ x, CGRing ring, int count, Dims4 d, BoxDecoder bx, uint32_t nint,
           const CGState *st) {
  pdl_wait();
  pdl_launch_dependents();
  float al[CG_RING];
#pragma unroll
  for (int m = 0; m < CG_RING; ++m) al[m] = st->al[m];
  for (uint32_t n = blockIdx.x * blockDim.x + threadIdx.x; n < nint; n += gridDim.x * blockDim.x) {
    int i, j, k, l;
    bx.decode(n, i, j, k, l);
    const idx_t id = d.index(i, j, k, l);
    float4 xx = x[id], t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int m = CG_RING - 2; m >= 0; --m)
      if (m < count) axpy4(t, al[m], __ldg(ring.p[m] + id));
    x[id] = make_float4(xx.x + t.x, xx.y + t.y, xx.z + t.z, xx.w + t.w);
  }
}

// Blocks per SM for a grid-stride PCG kernel: the tuned count, capped at what
// fits at once, so that the grid is a single wave.
template <class K>
int resident_per_sm(K kernel, int want) {
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, NT, 0) != cudaSuccess) {
    cudaGetLastError();
    n = 1;
  }
  if (n < 1) n = 1;
  return want < n ? want : n;
}

template <int NX, bool FILL, class GS>
void step_launch(float4 *x, float4 *r, const float4 *q, const CGRing &ring, int slot, GS gs,
                 Dims4 d, OFConsts c, CGState *st, double *dpart, float *fpart, int maxIter,
                 cudaStream_t s, const CGTune &tu) {
  static const int occ = resident_per_sm(k_cg_step<NX, FILL, GS>, 1 << 30);
  const long long n = interior_count(d);
  launch_pdl(k_cg_step<NX, FILL, GS>,
             grid_for(n > 0 ? n : 1, NT, tu.per_sm < occ ? tu.per_sm : occ), NT, s, x, r, q, ring,
             (const float4 *)ring.p[slot], ring.p[NX > 0 ? 0 : slot + 1], gs, d, interior_decoder(d),
             make_decoder(d.y, d.z, d.t, 0, 0, 0, 0), (uint32_t)n, c, st, dpart, fpart, maxIter);
}
template <class GS>
void step_any(float4 *x, float4 *r, const float4 *q, const CGRing &ring, int iter, GS gs, Dims4 d,
              OFConsts c, CGState *st, double *dpart, float *fpart, int maxIter, cudaStream_t s,
              const CGTune &tu) {
  const int slot = iter % ring.n;
  if (ring.n == 1)
    step_launch<1, false>(x, r, q, ring, slot, gs, d, c, st, dpart, fpart, maxIter, s, tu);
  else if (slot == CG_RING - 1)
    step_launch<CG_RING, false>(x, r, q, ring, slot, gs, d, c, st, dpart, fpart, maxIter, s, tu);
  else if (iter < CG_RING - 1)
    step_launch<0, true>(x, r, q, ring, slot, gs, d, c, st, dpart, fpart, maxIter, s, tu);
  else
    step_launch<0, false>(x, r, q, ring, slot, gs, d, c, st, dpart, fpart, maxIter, s, tu);
}
void launch_cg_step(float4 *x, float4 *r, const float4 *q, const CGRing &ring, int iter,
                    const float4 *g, const float *i1, Dims4 d, OFConsts c, CGState *st,
                    double *dpart, float *fpart, int maxIter, cudaStream_t s, const CGTune &tu) {
  if (i1)
    step_any(x, r, q, ring, iter, GradFromI1{i1, d.x, d.sz(), d.st(), c.dxf}, d, c, st, dpart,
             fpart, maxIter, s, tu);
  else
    step_any(x, r, q, ring, iter, GradStored<float4>{g}, d, c, st, dpart, fpart, maxIter, s, tu);
}
void launch_cg_step(float4 *x, float4 *r, const float4 *q, const CGRing &ring, int iter,
                    const BF4 *g, const float *, Dims4 d, OFConsts c, CGState *st, double *dpart,
                    float *fpart, int maxIter, cudaStream_t s, const CGTune &tu) {
  step_any(x, r, q, ring, iter, GradStored<BF4>{g}, d, c, st, dpart, fpart, maxIter, s, tu);
}
void launch_cg_flush(float4 *x, const CGRing &ring, int count, Dims4 d, CGState *st,
                     cudaStream_t s) {
  const long long n = interior_count(d);
  launch_pdl(k_cg_flush, grid_for(n > 0 ? n : 1, NT), NT, s, x, ring, count, d,
             interior_decoder(d), (uint32_t)n, (const CGState *)st);
}

// vel = x / mDx (optflow4d.cpp:520-529); a NaN residual resets the result to
// zero first (:508-514).
__global__ void k_of_copy_back(const float4 *__restrict__ x, float4 *__restrict__ vel,
                               long long n, float mDx, const CGState *st) {
  const float res = st->retResidual;
  const bool reset = (res != res);
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
       q += (long long)gridDim.x * blockDim.x) {
    float4 v = reset ? make_float4(0.f, 0.f, 0.f, 0.f) : __ldg(x + q);
    v.x = v.x / mDx;
    v.y = v.y / mDx;
    v.z = v.z / mDx;
    v.w = v.w / mDx;
    vel[q] = v;
  }
}
void launch_of_copy_back(const float4 *x, float4 *vel, long long cells,
                         float mDx, const CGState *st, cudaStream_t s) {
  k_of_copy_back<<<grid_for(cells, NT), NT, 0, s>>>(x, vel, cells, mDx, st);
}

// ---------------------------------------------------------------------------
// Gaussian blur (knGaussianBlur, optflow4d.cpp:132-158)
// ---------------------------------------------------------------------------

struct WTab {
  float w[160];  // exp weight by squared tap distance, s <= 6
};

template <int NC>
__global__ void __launch_bounds__(NT)
k_gauss_pass(const float *__restrict__ src, float *__restrict__ dst, Dims4 d,
             BoxDecoder bx, int s, WTab wt, int zero_border) {
  const uint32_t n = (uint32_t)d.cells();
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < n;
       q += gridDim.x * blockDim.x) {
    int i, j, k, l;
    bx.decode(q, i, j, k, l);
    if (!in_bounds(d, i, j, k, l, 1)) {
      if (zero_border) {
        if (NC == 4) ((float4 *)dst)[q] = make_float4(0.f, 0.f, 0.f, 0.f);
        else dst[q] = 0.f;
      }
      continue;
    }
    float4 val = make_float4(0.f, 0.f, 0.f, 0.f);
    float weight = 0.f;
    for (int vt = l - s; vt <= l + s; vt++) {
      if (vt < 0 || vt >= d.t) continue;
      for (int zk = k - s; zk <= k + s; zk++) {
        if (zk < 0 || zk >= d.z) continue;
        for (int yj = j - s; yj <= j + s; yj++) {
          if (yj < 0 || yj >= d.y) continue;
          const int base = (vt - l) * (vt - l) + (zk - k) * (zk - k) + (yj - j) * (yj - j);
          const idx_t row = d.index(0, yj, zk, vt);
          for (int xi = i - s; xi <= i + s; xi++) {
            if (xi < 0 || xi >= d.x) continue;
            const float w = wt.w[base + (xi - i) * (xi - i)];
            weight += w;
            if (NC == 4) {
              const float4 a = __ldg((const float4 *)src + row + xi);
              val.x += w * a.x;
              val.y += w * a.y;
              val.z += w * a.z;
              val.w += w * a.w;
            } else {
              val.x += w * __ldg(src + row + xi);
            }
          }
        }
      }
    }
    if (weight > 1e-6f) {
      if (NC == 4)
        ((float4 *)dst)[q] = make_float4(val.x / weight, val.y / weight, val.z / weight,
                                         val.w / weight);
      else
        dst[q] = val.x / weight;
    } else {
      if (NC == 4) ((float4 *)dst)[q] = __ldg((const float4 *)src + q);
      else dst[q] = __ldg(src + q);
    }
  }
}

void launch_gauss_pass(const float *src, float *dst, Dims4 d, int nc, int s,
                       const float *wtab, int zero_border, cudaStream_t st) {
  WTab wt;
  const int nw = 4 * s * s + 1;
  for (int q = 0; q < 160; ++q) wt.w[q] = q < nw ? wtab[q] : 0.f;
  BoxDecoder bx = make_decoder(d.x, d.y, d.z, 0, 0, 0, 0);
  const int nb = grid_for(d.cells(), NT, 8);
  if (nc == 4)
    k_gauss_pass<4><<<nb, NT, 0, st>>>(src, dst, d, bx, s, wt, zero_border);
  else
    k_gauss_pass<1><<<nb, NT, 0, st>>>(src, dst, d, bx, s, wt, zero_border);
}

// The separable blur (blurType 2).  Along one axis, the sum at coordinate c
// is sum_o w|o| src(c + o) over the in-range taps o = -S..S in increasing o,
// each added by one fused multiply-add, times 1 / (the in-range weights
// added in the same order): the 1D normalised Gaussian with clipping.  The
// four axes are applied in the order x, y, z, t by two kernels: one forms
// the y sums of x sums within each (z, t) plane, the other the t sums of z
// sums, each thread walking a run of y rows or t planes with the 2S + 1
// inner sums it needs in a register ring.  Every intermediate value is the
// single-axis pass's, rounded once to float, so the pair equals four
// single-axis passes; the 4D weight of the reference's blur is the product
// of the 1D weights and its in-bounds box the product of the 1D ranges, so
// the result equals the direct normalised stencil up to rounding.
struct W1 {
  float w[7];  // 1D weight by tap distance, S <= 6
};
template <int NC>
__device__ __forceinline__ float4 ld_nc(const float *p, idx_t i) {
  if (NC == 4) return __ldg((const float4 *)p + i);
  return make_float4(__ldg(p + i), 0.f, 0.f, 0.f);
}
template <int NC>
__device__ __forceinline__ void st_nc(float *p, idx_t i, float4 v) {
  if (NC == 4) ((float4 *)p)[i] = v;
  else p[i] = v.x;
}
__device__ __forceinline__ void fma4(float4 &v, float w, const float4 &a) {
  v.x = __fmaf_rn(w, a.x, v.x);
  v.y = __fmaf_rn(w, a.y, v.y);
  v.z = __fmaf_rn(w, a.z, v.z);
  v.w = __fmaf_rn(w, a.w, v.w);
}
__device__ __forceinline__ float4 scale4(const float4 &v, float s) {
  return make_float4(v.x * s, v.y * s, v.z * s, v.w * s);
}
// 1 / (sum of the in-range 1D weights around c on an axis of n cells)
template <int S>
__device__ __forceinline__ float sep_inv(const W1 &w, int c, int n) {
  float weight = 0.f;
#pragma unroll
  for (int o = -S; o <= S; ++o)
    if (c + o >= 0 && c + o < n) weight += w.w[o < 0 ? -o : o];
  return 1.0f / weight;
}
// the normalised 1D sum of the ring r (values at c - S .. c + S)
template <int S>
__device__ __forceinline__ float4 sep_ring(const W1 &w, const float4 (&r)[2 * S + 1], int c, int n) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int o = -S; o <= S; ++o)
    if (c + o >= 0 && c + o < n) fma4(v, w.w[o < 0 ? -o : o], r[o + S]);
  return scale4(v, sep_inv<S>(w, c, n));
}

constexpr int SEP_RUN = 16;  // y rows or t planes walked per thread
constexpr int SEP_ZB = 8;    // z planes per block of the z-t kernel (32 x 8 threads)
static_assert(32 * SEP_ZB == NT, "the z-t kernel's block is NT threads");

// The 2S + 1 taps of an axis sum around cell `id` with stride `step`; taps
// outside the axis (c + o out of 0..n-1) or a cell outside the walk
// (live == false) read as zero and are never used.
template <int NC, int S>
__device__ __forceinline__ void load_taps(float4 (&a)[2 * S + 1], const float *src, idx_t id,
                                          idx_t step, int c, int n, bool live) {
#pragma unroll
  for (int o = -S; o <= S; ++o)
    a[o + S] = (live && c + o >= 0 && c + o < n) ? ld_nc<NC>(src, id + o * step)
                                                 : make_float4(0.f, 0.f, 0.f, 0.f);
}
template <int S>
__device__ __forceinline__ float4 sum_taps(const W1 &w, const float4 (&a)[2 * S + 1], int c, int n,
                                           float inv) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int o = -S; o <= S; ++o)
    if (c + o >= 0 && c + o < n) fma4(v, w.w[o < 0 ? -o : o], a[o + S]);
  return scale4(v, inv);
}

// dst(x, y, z, t) = the y sum of the x sums, every cell of the box.  A thread walks a
// run of y rows; the taps of the next row are loaded before the current
// row's sums are formed.
template <int NC, int S>
__global__ void __launch_bounds__(NT)
k_blur_sep_xy(const float *__restrict__ src, float *__restrict__ dst, Dims4 d, W1 w, CellBox box,
              uint32_t n) {
  const idx_t sY = d.x;
  const uint32_t ex = box.hi[0] - box.lo[0], ez = box.hi[2] - box.lo[2], et = box.hi[3] - box.lo[3];
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    const int x = box.lo[0] + (int)(q % ex);
    uint32_t r = q / ex;
    const int z = box.lo[2] + (int)(r % ez);
    r /= ez;
    const int t = box.lo[3] + (int)(r % et);
    const int ya = box.lo[1] + (int)(r / et) * SEP_RUN, yb = min(ya + SEP_RUN, box.hi[1]);
    const idx_t plane = d.index(x, 0, z, t);
    const float ix = sep_inv<S>(w, x, d.x);
    float4 ring[2 * S + 1], a[2 * S + 1];
#pragma unroll
    for (int k = 1; k <= 2 * S; ++k) {
      const int y = ya - S - 1 + k;
      const bool live = y >= 0 && y < d.y;
      load_taps<NC, S>(a, src, plane + y * sY, 1, x, d.x, live);
      ring[k] = sum_taps<S>(w, a, x, d.x, ix);
    }
    load_taps<NC, S>(a, src, plane + (ya + S) * sY, 1, x, d.x, ya + S < d.y);
    for (int y = ya; y < yb; ++y) {
      float4 cur[2 * S + 1];
#pragma unroll
      for (int k = 0; k <= 2 * S; ++k) cur[k] = a[k];
      load_taps<NC, S>(a, src, plane + (y + S + 1) * sY, 1, x, d.x, y + 1 < yb && y + S + 1 < d.y);
#pragma unroll
      for (int k = 0; k < 2 * S; ++k) ring[k] = ring[k + 1];
      ring[2 * S] = sum_taps<S>(w, cur, x, d.x, ix);
      st_nc<NC>(dst, plane + y * sY, sep_ring<S>(w, ring, y, d.y));
    }
  }
}

// dst(x, y, z, t) = the t sum of the z sums at the box's interior cells; border_mode 1
// writes zeros on the one-cell ring, 2 leaves it alone.  A block is 32 x
// columns by SEP_ZB z planes at one y, so the z taps of a thread are mostly
// its neighbours' cells, read through L1; each thread walks a run of t
// planes, loading the next plane's taps before the current sums are formed.
template <int NC, int S>
__global__ void __launch_bounds__(NT)
k_blur_sep_zt(const float *__restrict__ src, float *__restrict__ dst, Dims4 d, W1 w,
              int border_mode, CellBox box, int xtiles, int ztiles, uint32_t nblocks) {
  const idx_t sZ = d.sz(), sT = d.st();
  const uint32_t ey = box.hi[1] - box.lo[1];
  const int tx = threadIdx.x & 31, tz = threadIdx.x >> 5;
  for (uint32_t b = blockIdx.x; b < nblocks; b += gridDim.x) {
    uint32_t r = b;
    const int xt = (int)(r % (uint32_t)xtiles);
    r /= (uint32_t)xtiles;
    const int y = box.lo[1] + (int)(r % ey);
    r /= ey;
    const int zt = (int)(r % (uint32_t)ztiles);
    const int ta = box.lo[3] + (int)(r / (uint32_t)ztiles) * SEP_RUN, tb = min(ta + SEP_RUN, box.hi[3]);
    const int x = box.lo[0] + xt * 32 + tx, z = box.lo[2] + zt * SEP_ZB + tz;
    if (x >= box.hi[0] || z >= box.hi[2]) continue;
    const idx_t col = d.index(x, y, z, 0);
    const bool ring_xyz = x < 1 || x >= d.x - 1 || y < 1 || y >= d.y - 1 || z < 1 || z >= d.z - 1;
    if (ring_xyz) {
      if (border_mode == 1)
        for (int t = ta; t < tb; ++t) st_nc<NC>(dst, col + t * sT, make_float4(0.f, 0.f, 0.f, 0.f));
      continue;
    }
    const float iz = sep_inv<S>(w, z, d.z);
    float4 ring[2 * S + 1], a[2 * S + 1];
#pragma unroll
    for (int k = 1; k <= 2 * S; ++k) {
      const int t = ta - S - 1 + k;
      load_taps<NC, S>(a, src, col + t * sT, sZ, z, d.z, t >= 0 && t < d.t);
      ring[k] = sum_taps<S>(w, a, z, d.z, iz);
    }
    load_taps<NC, S>(a, src, col + (ta + S) * sT, sZ, z, d.z, ta + S < d.t);
    for (int t = ta; t < tb; ++t) {
      float4 cur[2 * S + 1];
#pragma unroll
      for (int k = 0; k <= 2 * S; ++k) cur[k] = a[k];
      load_taps<NC, S>(a, src, col + (t + S + 1) * sT, sZ, z, d.z, t + 1 < tb && t + S + 1 < d.t);
#pragma unroll
      for (int k = 0; k < 2 * S; ++k) ring[k] = ring[k + 1];
      ring[2 * S] = sum_taps<S>(w, cur, z, d.z, iz);
      if (t < 1 || t >= d.t - 1) {
        if (border_mode == 1) st_nc<NC>(dst, col + t * sT, make_float4(0.f, 0.f, 0.f, 0.f));
        continue;
      }
      st_nc<NC>(dst, col + t * sT, sep_ring<S>(w, ring, t, d.t));
    }
  }
}

template <int NC, int S>
void launch_sep_pair(const float *src, float *dst, Dims4 d, int zt, const W1 &w, int border_mode,
                     const CellBox &box, cudaStream_t st) {
  const long long ex = box.hi[0] - box.lo[0], ey = box.hi[1] - box.lo[1],
                  ez = box.hi[2] - box.lo[2], et = box.hi[3] - box.lo[3];
  if (!zt) {
    const uint32_t n = (uint32_t)(ex * ez * et * ((ey + SEP_RUN - 1) / SEP_RUN));
    k_blur_sep_xy<NC, S><<<grid_for(n, NT, 8), NT, 0, st>>>(src, dst, d, w, box, n);
  } else {
    const int xtiles = (int)(ex + 31) / 32, ztiles = (int)(ez + SEP_ZB - 1) / SEP_ZB;
    const uint32_t nb = (uint32_t)(xtiles * ey * ztiles * ((et + SEP_RUN - 1) / SEP_RUN));
    const int grid = (int)std::min<long long>(nb, (long long)sm_count() * 8);
    k_blur_sep_zt<NC, S><<<grid, 32 * SEP_ZB, 0, st>>>(src, dst, d, w, border_mode, box, xtiles,
                                                       ztiles, nb);
  }
}
template <int NC>
void launch_sep_pair_nc(const float *src, float *dst, Dims4 d, int zt, int s, const W1 &w,
                        int border_mode, const CellBox &box, cudaStream_t st) {
  switch (s) {
    case 1: launch_sep_pair<NC, 1>(src, dst, d, zt, w, border_mode, box, st); break;
    case 2: launch_sep_pair<NC, 2>(src, dst, d, zt, w, border_mode, box, st); break;
    case 3: launch_sep_pair<NC, 3>(src, dst, d, zt, w, border_mode, box, st); break;
    case 4: launch_sep_pair<NC, 4>(src, dst, d, zt, w, border_mode, box, st); break;
    case 5: launch_sep_pair<NC, 5>(src, dst, d, zt, w, border_mode, box, st); break;
    default: launch_sep_pair<NC, 6>(src, dst, d, zt, w, border_mode, box, st); break;
  }
}

void launch_gauss_sep_pair(const float *src, float *dst, Dims4 d, int nc, int zt, int s,
                           const float *w1d, int border_mode, const CellBox &box,
                           cudaStream_t st) {
  if (box.cells() == 0) return;
  W1 w;
  for (int q = 0; q < 7; ++q) w.w[q] = q <= s ? w1d[q] : 0.f;
  if (nc == 4) launch_sep_pair_nc<4>(src, dst, d, zt, s, w, border_mode, box, st);
  else launch_sep_pair_nc<1>(src, dst, d, zt, s, w, border_mode, box, st);
}

// ---------------------------------------------------------------------------
// Projection correction (optflow4d.cpp:651-734)
// ---------------------------------------------------------------------------

// The projection samples phiOrg 9 times around each cell (the centre and
// +-0.5 along each axis for the normal) and then once per search step.  The
// samples share taps: along each axis the +-0.5 bases differ from the
// centre's by at most one, so the 2^4 centre block plus one 8-tap face per
// shifted sample that moved covers all nine (48 loads instead of 144 when
// nothing is clamped).  Search steps reuse the taps while the probe stays in
// the same cell, which is every step once the normal is zero (flat, clamped
// regions).  The weights and the sum order are those of interp4_real, so the
// values are the same bit for bit.

// c[t*8 + z*4 + x*2 + y]: the interp4_sum order.
__device__ __forceinline__ float ip16(const float (&c)[16], const AxisW &ax, const AxisW &ay,
                                      const AxisW &az, const AxisW &at) {
  const float s0 = ax.w0, s1 = ax.w1, t0 = ay.w0, t1 = ay.w1;
  const float f0 = az.w0, f1 = az.w1, g0 = at.w0, g1 = at.w1;
  return (((c[0] * t0 + c[1] * t1) * s0 + (c[2] * t0 + c[3] * t1) * s1) * f0 +
          ((c[4] * t0 + c[5] * t1) * s0 + (c[6] * t0 + c[7] * t1) * s1) * f1) *
             g0 +
         (((c[8] * t0 + c[9] * t1) * s0 + (c[10] * t0 + c[11] * t1) * s1) * f0 +
          ((c[12] * t0 + c[13] * t1) * s0 + (c[14] * t0 + c[15] * t1) * s1) * f1) *
             g1;
}

__device__ __forceinline__ idx_t tap_off(int q, idx_t sY, idx_t sZ, idx_t sT) {
  return (idx_t)((q >> 1) & 1) + (idx_t)(q & 1) * sY + (idx_t)((q >> 2) & 1) * sZ +
         (idx_t)((q >> 3) & 1) * sT;
}

__device__ __forceinline__ void load_taps(const float *__restrict__ phi, idx_t i, idx_t sY,
                                          idx_t sZ, idx_t sT, float (&c)[16]) {
#pragma unroll
  for (int q = 0; q < 16; ++q) c[q] = __ldg(phi + i + tap_off(q, sY, sZ, sT));
}

// The sample at the centre position with axis D moved to `s`.
template <int D>
__device__ __forceinline__ float shifted_sample(const float *__restrict__ phi, const Dims4 &d,
                                                const float (&C)[16], idx_t ic,
                                                const AxisW (&a)[4], const AxisW &s, float p0,
                                                float p1, float p2, float p3) {
  constexpr int bit = D == 0 ? 2 : D == 1 ? 1 : D == 2 ? 4 : 8;
  const idx_t sY = d.x, sZ = d.sz(), sT = d.st();
  const idx_t sD = D == 0 ? 1 : D == 1 ? sY : D == 2 ? sZ : sT;
  const int delta = s.b - a[D].b;
  if (delta < -1 || delta > 1) return interp4_real(phi, d, p0, p1, p2, p3);
  float S[16];
  if (delta == 0) {
#pragma unroll
    for (int q = 0; q < 16; ++q) S[q] = C[q];
  } else if (delta > 0) {
    const idx_t f = ic + 2 * sD;
#pragma unroll
    for (int q = 0; q < 16; ++q)
      if (!(q & bit)) {
        S[q] = C[q | bit];
        S[q | bit] = __ldg(phi + f + tap_off(q, sY, sZ, sT));
      }
  } else {
    const idx_t f = ic - sD;
#pragma unroll
    for (int q = 0; q < 16; ++q)
      if (!(q & bit)) {
        S[q] = __ldg(phi + f + tap_off(q, sY, sZ, sT));
        S[q | bit] = C[q];
      }
  }
  return ip16(S, D == 0 ? s : a[0], D == 1 ? s : a[1], D == 2 ? s : a[2], D == 3 ? s : a[3]);
}

// The state of a cell whose projection search is still to run.
struct ProjState {
  float4 p;    // the advected position
  float4 nrm;  // the normalised normal
  float dd, target;
  uint32_t id, pad;
};

// The outcome of a cell's projection (optflow4d.cpp:725-732): dst, dst2 (the
// extrapolation's second buffer, nullable) and marker stay zero where the
// distance found is above the threshold.
__device__ __forceinline__ void project_write(float4 *__restrict__ dst, float4 *__restrict__ dst2,
                                              float *__restrict__ marker, idx_t id, float4 nrm,
                                              float dd, float threshPhi) {
  if (fabsf(dd) > threshPhi) return;
  const float4 v = make_float4(nrm.x * dd, nrm.y * dd, nrm.z * dd, nrm.w * dd);
  dst[id] = v;
  if (dst2) dst2[id] = v;
  marker[id] = 1.f;
}

// knProjectCells, first part: per box cell the advected position, the normal
// and the start of the search.  Cells with a zero normal (flat, clamped phi)
// finish here; the others are appended to `queue` (warp-aggregated, in no
// fixed order) for k_project_search.
// One trip per thread: a capped grid of 16 blocks per SM with 5 or 6 resident
// ended in a mostly empty wave (64^4: 808 us with 5 blocks of 96 registers and
// that grid, 729 with the blocks refilled as they end, 690 with 6 blocks per SM;
// 8 per SM 696).
__global__ void __launch_bounds__(128, 6)
k_project_prep(float4 *__restrict__ dst, float4 *__restrict__ dst2,
               const float4 *__restrict__ vel,
               const float *__restrict__ phiOrg, const float *__restrict__ phiTarget,
               float *__restrict__ marker, Dims4 d, BoxDecoder bx, uint32_t nbox,
               float threshPhi, int maxIter, ProjState *__restrict__ queue,
               unsigned int *__restrict__ qcount) {
  const idx_t sY = d.x, sZ = d.sz(), sT = d.st();
  // every lane of a warp runs the same trip count, for the warp-wide append
  const uint32_t stride = gridDim.x * blockDim.x;
  const uint32_t trips = (nbox + stride - 1) / stride;
  const unsigned lane = threadIdx.x & 31;
  for (uint32_t it = 0, q = blockIdx.x * blockDim.x + threadIdx.x; it < trips; ++it, q += stride) {
    bool search = false;
    ProjState S;
    if (q < nbox) {
    int i, j, k, l;
    bx.decode(q, i, j, k, l);
    const idx_t id = d.index(i, j, k, l);
    const float dt = 1.0f;
    const float4 v = __ldg(vel + id);
    const float p0 = (float)(i + 0.5f) - v.x * dt;
    const float p1 = (float)(j + 0.5f) - v.y * dt;
    const float p2 = (float)(k + 0.5f) - v.z * dt;
    const float p3 = (float)(l + 0.5f) - v.w * dt;
    const AxisW a[4] = {axis_index(p0, d.x), axis_index(p1, d.y), axis_index(p2, d.z),
                        axis_index(p3, d.t)};
    const idx_t ic = d.index(a[0].b, a[1].b, a[2].b, a[3].b);
    float T[16];
    load_taps(phiOrg, ic, sY, sZ, sT, T);
    // normal at p: central differences with h = 0.5 (optflow4d.cpp:655-661)
    const float h = 0.5f;
    float4 nrm;
    nrm.x = shifted_sample<0>(phiOrg, d, T, ic, a, axis_index(p0 + h, d.x), p0 + h, p1, p2, p3) -
            shifted_sample<0>(phiOrg, d, T, ic, a, axis_index(p0 - h, d.x), p0 - h, p1, p2, p3);
    nrm.y = shifted_sample<1>(phiOrg, d, T, ic, a, axis_index(p1 + h, d.y), p0, p1 + h, p2, p3) -
            shifted_sample<1>(phiOrg, d, T, ic, a, axis_index(p1 - h, d.y), p0, p1 - h, p2, p3);
    nrm.z = shifted_sample<2>(phiOrg, d, T, ic, a, axis_index(p2 + h, d.z), p0, p1, p2 + h, p3) -
            shifted_sample<2>(phiOrg, d, T, ic, a, axis_index(p2 - h, d.z), p0, p1, p2 - h, p3);
    nrm.w = shifted_sample<3>(phiOrg, d, T, ic, a, axis_index(p3 + h, d.t), p0, p1, p2, p3 + h) -
            shifted_sample<3>(phiOrg, d, T, ic, a, axis_index(p3 - h, d.t), p0, p1, p2, p3 - h);
    // normalize (util/vector4d.h:331-345)
    {
      // |len2 - 1| < 1e-12 in double holds for a float len2 only at 1.0f:
      // the floats next to 1 are 2^-24 and 2^-23 away.  The float test keeps
      // the FP64 pipe (2 ops/clk/SM on this part) out of the kernel.
      const float len2 = nrm.x * nrm.x + nrm.y * nrm.y + nrm.z * nrm.z + nrm.w * nrm.w;
      const float eps2 = 1e-6f * 1e-6f;
      if (len2 == 1.0f) {
        // normalized enough
      } else if (len2 > eps2) {
        const float nl = __fsqrt_rn(len2);
        const float inv = __frcp_rn(nl);
        nrm.x *= inv;
        nrm.y *= inv;
        nrm.z *= inv;
        nrm.w *= inv;
      } else {
        nrm = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    // projectCell (optflow4d.cpp:675-710)
    float step = 0.25f;
    if (maxIter < 50) step = 0.5f;
    const float targetVal = __ldg(phiTarget + id);
    const float vn = ip16(T, a[0], a[1], a[2], a[3]);
    float dd = (vn - targetVal);
    if (nrm.x == 0.f && nrm.y == 0.f && nrm.z == 0.f && nrm.w == 0.f && isfinite(dd)) {
      // Zero normal (flat, clamped phi): every probe is p itself (p + 0 * dd),
      // so vn and the in-bounds test never change, the direction never flips,
      // the step never halves and the loop runs maxIter plain steps.
      if (maxIter > 0) {
        if (!in_bounds(d, trunc_i(p0), trunc_i(p1), trunc_i(p2), trunc_i(p3), 0)) {
          dd = 9999.f;
        } else if (vn < targetVal) {
          for (int s = 0; s < maxIter; ++s) dd += step;
        } else {
          for (int s = 0; s < maxIter; ++s) dd -= step;
        }
      }
      project_write(dst, dst2, marker, id, nrm, dd, threshPhi);
    } else if (maxIter <= 0) {
      project_write(dst, dst2, marker, id, nrm, dd, threshPhi);
    } else {
      search = true;
      S.p = make_float4(p0, p1, p2, p3);
      S.nrm = nrm;
      S.dd = dd;
      S.target = targetVal;
      S.id = (uint32_t)id;
      S.pad = 0;
    }
    }
    const unsigned want = __ballot_sync(0xffffffffu, search);
    if (want) {
      unsigned base = 0;
      if (lane == (unsigned)(__ffs(want) - 1)) base = atomicAdd(qcount, (unsigned)__popc(want));
      base = __shfl_sync(0xffffffffu, base, __ffs(want) - 1);
      if (search) queue[base + __popc(want & ((1u << lane) - 1u))] = S;
    }
  }
}

// knProjectCells, the search (projectCell, optflow4d.cpp:675-710) of the
// queued cells.  A lane pulls its next cell when its search ends, so the
// lanes of a warp stay busy whatever the cells' step counts (1 to maxIter).
// Warps take chunks of PROJ_CHUNK queue entries; within a chunk the lanes
// that need a cell take consecutive entries in lane order.  Every cell's
// arithmetic is the single-cell search's, so the results do not depend on
// which lane runs a cell.
constexpr int PROJ_CHUNK = 64;
__global__ void __launch_bounds__(128)
k_project_search(float4 *__restrict__ dst, float4 *__restrict__ dst2,
                 const float *__restrict__ phiOrg,
                 float *__restrict__ marker, Dims4 d, float threshPhi, int maxIter,
                 const ProjState *__restrict__ queue, const unsigned int *__restrict__ qcount,
                 unsigned int *__restrict__ qhead) {
  const idx_t sY = d.x, sZ = d.sz(), sT = d.st();
  const unsigned lane = threadIdx.x & 31;
  const unsigned n = *qcount;
  const float dt = 1.0f;
  unsigned next = 0, end = 0;  // the warp's current chunk
  bool drained = false;        // the queue has no chunk left for this warp
  bool active = false;
  ProjState S;
  float T[16];
  idx_t ti = -1;
  float step = 0.f;
  int lastDir = 0, s = 0;
  for (;;) {
    unsigned need = __ballot_sync(0xffffffffu, !active);
    while (need && !drained) {
      if (next >= end) {
        unsigned base = 0;
        if (lane == 0) base = atomicAdd(qhead, (unsigned)PROJ_CHUNK);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= n) {
          drained = true;
          break;
        }
        next = base;
        end = min(base + (unsigned)PROJ_CHUNK, n);
      }
      const unsigned k = next + __popc(need & ((1u << lane) - 1u));
      if (!active && k < end) {
        S = queue[k];
        active = true;
        ti = -1;
        step = maxIter < 50 ? 0.5f : 0.25f;
        lastDir = 0;
        s = 0;
      }
      next = min(next + (unsigned)__popc(need), end);
      need = __ballot_sync(0xffffffffu, !active);
    }
    if (!__any_sync(0xffffffffu, active)) break;
    if (active) {
    // one step of the search
    bool done = false;
    const float n0 = S.p.x + (S.nrm.x * S.dd) * dt;
    const float n1 = S.p.y + (S.nrm.y * S.dd) * dt;
    const float n2 = S.p.z + (S.nrm.z * S.dd) * dt;
    const float n3 = S.p.w + (S.nrm.w * S.dd) * dt;
    if (!in_bounds(d, trunc_i(n0), trunc_i(n1), trunc_i(n2), trunc_i(n3), 0)) {
      S.dd = 9999.f;
      done = true;
    } else {
      const AxisW b0 = axis_index(n0, d.x), b1 = axis_index(n1, d.y);
      const AxisW b2 = axis_index(n2, d.z), b3 = axis_index(n3, d.t);
      const idx_t ni = d.index(b0.b, b1.b, b2.b, b3.b);
      if (ni != ti) {
        load_taps(phiOrg, ni, sY, sZ, sT, T);
        ti = ni;
      }
      const float vn = ip16(T, b0, b1, b2, b3);
      if (vn < S.target) {
        if (lastDir < 0) step *= 0.5f;
        S.dd += step;
        lastDir = 1;
      } else {
        if (lastDir > 0) step *= 0.5f;
        S.dd -= step;
        lastDir = -1;
      }
      // (double)step < 0.1 equals step < 0.1f for every float: 0.1f is the
      // smallest float above 0.1.
      if (step < 0.1f) done = true;
    }
    if (++s >= maxIter) done = true;
    if (done) {
      project_write(dst, dst2, marker, S.id, S.nrm, S.dd, threshPhi);
      active = false;
    }
    }
  }
}

__global__ void k_zero_counters(unsigned int *c) {
  c[0] = 0;
  c[1] = 0;
}

// Queue entries: the whole box, or at least PROJ_QMIN cells and a quarter of
// the box, whichever is less; a larger box runs in t slabs of that many
// cells.
constexpr long long PROJ_QMIN = 16ll << 20;
long long project_queue_cells(Dims4 d) {
  if (d.x < 5 || d.y < 5 || d.z < 5 || d.t < 5) return 1;
  const long long vol = (long long)(d.x - 4) * (d.y - 4) * (d.z - 4);
  const long long nbox = vol * (d.t - 4);
  long long cap = nbox / 4 > PROJ_QMIN ? nbox / 4 : PROJ_QMIN;
  if (cap < vol) cap = vol;  // at least one t plane
  return cap < nbox ? cap : nbox;
}

size_t project_queue_bytes(Dims4 d) { return sizeof(ProjState) * (size_t)project_queue_cells(d); }

void launch_project_cells(float4 *dst, float4 *dst2, const float4 *vel, const float *phiOrg,
                          const float *phiTarget, float *marker, Dims4 d,
                          float threshPhi, int maxIter, void *queue, unsigned int *counters,
                          cudaStream_t s) {
  if (d.x < 5 || d.y < 5 || d.z < 5 || d.t < 5) return;
  const long long vol = (long long)(d.x - 4) * (d.y - 4) * (d.z - 4);
  const int tslab = (int)(project_queue_cells(d) / vol);  // t planes per slab
  // every block of the search resident at once: warps leave when the queue
  // is drained
  static const int per_sm = [] {
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_project_search, 128, 0);
    return n < 1 ? 1 : n;
  }();
  for (int t0 = 0; t0 < d.t - 4; t0 += tslab) {
    const int nt = min(tslab, d.t - 4 - t0);
    const BoxDecoder bx = make_decoder(d.x - 4, d.y - 4, d.z - 4, 2, 2, 2, 2 + t0);
    const long long nbox = vol * nt;
    if (t0 > 0) k_zero_counters<<<1, 1, 0, s>>>(counters);
    k_project_prep<<<(unsigned)((nbox + 127) / 128), 128, 0, s>>>(
        dst, dst2, vel, phiOrg, phiTarget, marker, d, bx, (uint32_t)nbox, threshPhi, maxIter,
        (ProjState *)queue, counters);
    k_project_search<<<sm_count() * per_sm, 128, 0, s>>>(dst, dst2, phiOrg, marker, d, threshPhi,
                                                         maxIter, (const ProjState *)queue,
                                                         counters, counters + 1);
  }
}

// knCvExpolBlur4d (optflow4d.cpp:613-626) fused with the preceding copy:
// unmarked interior cells get avg of the 3^4 neighbourhood, scaled by the
// double constant 1/81 and rounded back to float; others copy through.
__global__ void __launch_bounds__(NT)
k_expol_sweep(const float4 *__restrict__ in, float4 *__restrict__ out,
              const float *__restrict__ mark, Dims4 d, BoxDecoder bx) {
  const uint32_t n = (uint32_t)d.cells();
  const idx_t sY = d.x, sZ = d.sz(), sT = d.st();
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < n;
       q += gridDim.x * blockDim.x) {
    int i, j, k, l;
    bx.decode(q, i, j, k, l);
    if (!in_bounds(d, i, j, k, l, 1) || __ldg(mark + q) != 0.f) {
      out[q] = __ldg(in + q);
      continue;
    }
    float4 val = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int vt = -1; vt <= 1; ++vt)
      for (int zk = -1; zk <= 1; ++zk)
        for (int yj = -1; yj <= 1; ++yj) {
          const idx_t row = (idx_t)q + vt * sT + zk * sZ + yj * sY;
#pragma unroll
          for (int xi = -1; xi <= 1; ++xi) {
            const float4 a = __ldg(in + row + xi);
            val.x += a.x;
            val.y += a.y;
            val.z += a.z;
            val.w += a.w;
          }
        }
    out[q] = make_float4(mul_inv81(val.x), mul_inv81(val.y), mul_inv81(val.z), mul_inv81(val.w));
  }
}

void launch_expol_sweep(const float4 *in, float4 *out, const float *mark,
                        Dims4 d, cudaStream_t s) {
  BoxDecoder bx = make_decoder(d.x, d.y, d.z, 0, 0, 0, 0);
  k_expol_sweep<<<grid_for(d.cells(), NT, 8), NT, 0, s>>>(in, out, mark, d, bx);
}

}  // namespace flof
