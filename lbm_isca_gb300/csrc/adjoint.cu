// Adjoint kernels of the reference-layout time step: the transposes of
// lbm_tendency_grid (grid-point part of Dynamics.tendencies, reference
// dynamics.py:176-267) and of lbm_implicit_step (Integrator.step,
// integrator.py:264-315).  The spectral transforms need no kernels of their
// own: the transpose of each transform is another transform of the library
// with rescaled tables.  The column arithmetic lives in adjoint_col.cuh.
#include "lbm_common.cuh"
#include "adjoint_col.cuh"

namespace lbm {

// One thread per (column, level) and per (coefficient, level), ADJ_THREADS / K
// columns a block, the column's exchanges in shared memory.  Both are bound by the
// latency of a column's chain and the FP64 pipe: with one thread per column and
// its level arrays in local memory, one member of T42 filled 256 and 116 warps.
// At T42, 20 levels, one member, FP64: tendencies 239 -> 84 us, implicit update 146 -> 24.
constexpr int ADJ_THREADS = 256;

template <typename R>
__global__ void __launch_bounds__(ADJ_THREADS) k_tendency_grid_adj(lbm_tend_adj_args a) {
  const int J = a.nlat, I = a.nlon, K = a.kmax, CB = ADJ_THREADS / K;
  __shared__ R sgt[ADJ_THREADS], ske[ADJ_THREADS], ssa[ADJ_THREADS], ssb[ADJ_THREADS];
  __shared__ R spx[ADJ_THREADS], spy[ADJ_THREADS];
  const size_t ncol2 = (size_t)J * I;
  const int tid = threadIdx.x, cl = tid / K, k = tid - cl * K, cK = cl * K;
  const size_t col = (size_t)blockIdx.x * CB + cl;
  const bool act = cl < CB && col < (size_t)a.nmem * ncol2;
  const size_t ji = act ? col % ncol2 : 0;
  auto P = [](const void* p) { return (const R*)p; };
  const size_t b3 = ji * K, p3 = (act ? col : 0) * K;
  lbm_adj::ColConst<R> c;
  c.K = K;
  c.kappa = R(a.kappa);
  c.eps = R(a.epsvt);
  c.rair = R(a.rair);
  c.dsig = P(a.dsig);
  c.sigm = P(a.sigm);
  c.alpha = P(a.alpha);
  c.w3 = P(a.w3);
  c.wP = P(a.wP);
  c.cpg = P(a.cpg);
  c.ww = P(a.ww);
  c.tmtx = P(a.tmtx);
  c.tref = P(a.tref);
  c.ub = P(a.ub) + b3;
  c.vb = P(a.vb) + b3;
  c.tb = P(a.tb) + b3;
  c.qb = P(a.qb) + b3;
  c.tvb = P(a.tvb) + b3;
  c.absv = P(a.absvor) + b3;
  c.divb = P(a.divb) + b3;
  c.x5b = P(a.x5b) + b3;
  c.sdb = P(a.sdotb) + ji * (K + 1);
  c.pixb = P(a.pixb)[ji];
  c.piyb = P(a.piyb)[ji];
  c.u0 = a.u0 ? P(a.u0) + p3 : nullptr;
  c.v0 = a.v0 ? P(a.v0) + p3 : nullptr;
  const lbm_adj::TendAdjIn<R> y = {P(a.a_fu) + p3, P(a.a_fv) + p3, P(a.a_ke) + p3,
                                   P(a.a_gt) + p3, P(a.a_xu) + p3, P(a.a_xv) + p3,
                                   P(a.a_g) + p3,  P(a.a_yu) + p3, P(a.a_yv) + p3,
                                   act ? P(a.a_gt_pi)[col] : R(0)};
  if (act) {
    sgt[tid] = y.gt[k];
    ske[tid] = y.ke[k];
    lbm_adj::tendency_adj_sums(c, y, k, ssa + tid, ssb + tid);
  }
  __syncthreads();
  lbm_adj::TendAdjOut<R> o = {};
  if (act) {
    R cum = R(0);
    for (int l = 1; l < K; ++l) cum += ssb[cK + l];
    for (int l = 1; l <= k; ++l) cum += ssa[cK + l];
    o = lbm_adj::tendency_adj_level(c, y, k, cum, sgt + cK, ske + cK);
    spx[tid] = o.px;
    spy[tid] = o.py;
  }
  __syncthreads();                     // outputs may take the place of inputs
  if (act) {
    ((R*)a.a_u)[p3 + k] = o.u;
    ((R*)a.a_v)[p3 + k] = o.v;
    ((R*)a.a_t)[p3 + k] = o.t;
    ((R*)a.a_q)[p3 + k] = o.q;
    ((R*)a.a_vor)[p3 + k] = o.vor;
    ((R*)a.a_div)[p3 + k] = o.div;
  }
  // column sums: pi_x, then pi_y
  for (int x = tid; x < 2 * CB; x += ADJ_THREADS) {
    const int q = x % CB;
    const size_t cq = (size_t)blockIdx.x * CB + q;
    if (cq >= (size_t)a.nmem * ncol2) continue;
    const R* sp = (x < CB ? spx : spy) + q * K;
    R s = R(0);
    for (int l = 0; l < K; ++l) s += sp[l];
    ((R*)(x < CB ? a.a_pix : a.a_piy))[cq] = s;
  }
}

template <typename R>
__global__ void __launch_bounds__(ADJ_THREADS) k_implicit_adj(lbm_implicit_adj_args a) {
  using V = C2<R>;
  const int K = a.kmax, M = a.nmax + 1, CB = ADJ_THREADS / K;
  __shared__ V sh[4][ADJ_THREADS];
  const int tid = threadIdx.x, cl = tid / K, l = tid - cl * K, cK = cl * K;
  const size_t coef = (size_t)blockIdx.x * CB + cl;             // (e, m, n)
  const bool in = cl < CB && coef < (size_t)a.nmem * M * M;
  const int n = in ? (int)(coef % M) : 0, m = in ? (int)((coef / M) % M) : 0;
  const bool act = in && n >= m;
  const V z = cmk<R>(0, 0);
  const size_t o3 = (in ? coef : 0) * K + l, o2 = in ? coef : 0;
  auto P = [](const void* p) { return (const R*)p; };
  const void* an[4] = {a.an_vor, a.an_div, a.an_t, a.an_q};
  void* ap[4] = {a.ap_vor, a.ap_div, a.ap_t, a.ap_q};
  void* aw[4] = {a.aw_vor, a.aw_div, a.aw_t, a.aw_q};
  lbm_adj::ImplConst<R> c;
  c.K = K;
  c.dt = R(a.dt);
  c.lap = P(a.lap)[n];
  c.kv = P(a.kv) + (size_t)n * K;
  c.kd = P(a.kd) + (size_t)n * K;
  c.ktt = P(a.ktt) + (size_t)n * K;
  c.kq = P(a.kq) + (size_t)n * K;
  c.ww = P(a.ww);
  c.tmtx = P(a.tmtx);
  c.gg = P(a.gg);
  c.dsig = P(a.dsig);
  c.minv = P(a.minv) + (size_t)n * K * K;
  c.vd[0] = P(a.vd_vor);
  c.vd[1] = P(a.vd_div);
  c.vd[2] = P(a.vd_t);
  c.vd[3] = P(a.vd_q);
  c.vd_skip_vordiv = n < 2;
  const V anpi = act ? ((const V*)a.an_pi)[o2] : z;
  const V awpi = anpi * (R(2) * c.dt);
#pragma unroll
  for (int f = 0; f < 4; ++f) sh[f][tid] = act ? ((const V*)an[f])[o3] : z;
  __syncthreads();
  lbm_adj::ImplAdjLevel<V> o = {};
  if (act) {
    V v[4];
#pragma unroll
    for (int f = 0; f < 4; ++f) v[f] = lbm_adj::impl_adj_vdiff(c, f, sh[f] + cK, l, z);
    lbm_adj::impl_adj_point(c, l, v, o);
  }
  __syncthreads();
  sh[0][tid] = o.aw[2];
  __syncthreads();
  if (act) lbm_adj::impl_adj_dbar(c, l, sh[0] + cK, awpi, z, o);
  sh[1][tid] = o.x;
  __syncthreads();
  V part = z;
  if (act) part = lbm_adj::impl_adj_rhs(c, l, sh[1] + cK, z, o);
  sh[2][tid] = o.x;
  sh[3][tid] = part;
  __syncthreads();
  if (act) lbm_adj::impl_adj_wdx(c, l, sh[2] + cK, z, o);
  if (!in) return;
  // outside the triangle the update writes zeros
#pragma unroll
  for (int f = 0; f < 4; ++f) {
    ((V*)ap[f])[o3] = o.ap[f];
    ((V*)aw[f])[o3] = o.aw[f];
  }
  if (l == 0) {
    V s = z;
    for (int k = 0; k < K; ++k) s = s + sh[3][cK + k];
    ((V*)a.ap_pi)[o2] = anpi + s;
    ((V*)a.aw_pi)[o2] = awpi + s * c.dt;
  }
}

template <typename R>
static int tend_adj(const lbm_tend_adj_args* a, cudaStream_t st) {
  const size_t cols = (size_t)a->nmem * a->nlat * a->nlon, CB = ADJ_THREADS / a->kmax;
  k_tendency_grid_adj<R><<<(unsigned)((cols + CB - 1) / CB), ADJ_THREADS, 0, st>>>(*a);
  LBM_LAUNCH_CHECK();
  return LBM_OK;
}

template <typename R>
static int impl_adj(const lbm_implicit_adj_args* a, cudaStream_t st) {
  const size_t M = (size_t)a->nmax + 1, total = (size_t)a->nmem * M * M;
  const size_t CB = ADJ_THREADS / a->kmax;
  k_implicit_adj<R><<<(unsigned)((total + CB - 1) / CB), ADJ_THREADS, 0, st>>>(*a);
  LBM_LAUNCH_CHECK();
  return LBM_OK;
}

}  // namespace lbm

using namespace lbm;

extern "C" {

int lbm_tendency_grid_adjoint(int prec, const lbm_tend_adj_args* a, void* stream) {
  if (!a || a->nmem < 1 || a->kmax < 1 || a->kmax > 64 || a->nlat < 2 || a->nlon < 2)
    return LBM_ERR_ARG;
  const void* need[] = {a->dsig,  a->sigm, a->alpha, a->w3,    a->wP,    a->cpg,   a->ww,
                        a->tmtx,  a->tref, a->ub,    a->vb,    a->tb,    a->qb,    a->tvb,
                        a->absvor, a->divb, a->x5b,  a->sdotb, a->pixb,  a->piyb,  a->a_fu,
                        a->a_fv,  a->a_ke, a->a_gt,  a->a_xu,  a->a_xv,  a->a_g,   a->a_yu,
                        a->a_yv,  a->a_gt_pi, a->a_u, a->a_v,  a->a_t,   a->a_q,   a->a_vor,
                        a->a_div, a->a_pix, a->a_piy};
  for (const void* p : need)
    if (!p) return LBM_ERR_ARG;
  if ((a->u0 == nullptr) != (a->v0 == nullptr)) return LBM_ERR_ARG;
  if (prec == LBM_F64) return tend_adj<double>(a, (cudaStream_t)stream);
  if (prec == LBM_F32) return tend_adj<float>(a, (cudaStream_t)stream);
  return LBM_ERR_ARG;
}

int lbm_implicit_step_adjoint(int prec, const lbm_implicit_adj_args* a, void* stream) {
  if (!a || a->nmem < 1 || a->kmax < 1 || a->kmax > 64 || a->nmax < 1) return LBM_ERR_ARG;
  const void* need[] = {a->lap,    a->kv,     a->kd,    a->ktt,    a->kq,     a->ww,
                        a->tmtx,   a->gg,     a->dsig,  a->minv,   a->an_vor, a->an_div,
                        a->an_t,   a->an_pi,  a->an_q,  a->ap_vor, a->ap_div, a->ap_t,
                        a->ap_pi,  a->ap_q,   a->aw_vor, a->aw_div, a->aw_t,  a->aw_pi,
                        a->aw_q};
  for (const void* p : need)
    if (!p) return LBM_ERR_ARG;
  if (prec == LBM_F64) return impl_adj<double>(a, (cudaStream_t)stream);
  if (prec == LBM_F32) return impl_adj<float>(a, (cudaStream_t)stream);
  return LBM_ERR_ARG;
}

}  // extern "C"
