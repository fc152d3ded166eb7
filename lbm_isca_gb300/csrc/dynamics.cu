// Reference-layout kernels of the time step: the grid-point part of
// Dynamics.tendencies (dynamics.py:176-267) and Integrator.step
// (integrator.py:264-315).  The fused ensemble stepper (stepper.cu) runs the
// same algebra on its own layouts; these serve the drop-in API
// (Dynamics.tendencies / Integrator.step called directly, the forward
// start of LBM.run on an arbitrary grid state).
#include "lbm_common.cuh"

namespace lbm {

constexpr int KMAX_LOCAL = 64;   // largest level count the column kernels hold

// Vertical advection, SECOND_CENTERED ADVECTIVE_FORM with the overall +
// sign of dynamics.py:117-143: f(l) is a level accessor, s0 and s1 the
// vertical velocities at the half levels k and k + 1.
template <typename R, typename F>
LBM_D R vert_adv(int k, int K, F f, R s0, R s1, R dsk, R rdsk) {
  const R fk = f(k);
  const R flo = (k >= 1) ? s0 * R(0.5) * (fk + f(k - 1)) : R(0);
  const R fhi = (k + 1 <= K - 1) ? s1 * R(0.5) * (f(k + 1) + fk) : R(0);
  const R x = fhi - flo - fk * (s1 - s0);
  if constexpr (sizeof(R) == 8) return x * rdsk;   // a division costs ten products
  else return x / dsk;
}

// One thread per (column, level), TG_THREADS / K columns a block: consecutive
// lanes read consecutive levels, the column sums come from shared memory, each
// thread its own (the order of every sum is the level's).  Bound by the FP64 pipe
// (about 165 multiply-adds a level at 20 levels).  One thread per column
// with its level arrays in local memory left one member of T42 on 256 warps:
// 291 -> 83 us at T42, 20 levels, one member, FP64.
constexpr int TG_THREADS = 256;

template <typename R> size_t tend_smem(int K) {
  const int CB = TG_THREADS / K;
  return sizeof(R) * ((size_t)2 * K * K + 4 * (size_t)CB * K + CB);
}

template <typename R>
__global__ void __launch_bounds__(TG_THREADS) k_tendency_grid(lbm_tend_grid_args a) {
  const int J = a.nlat, I = a.nlon, K = a.kmax, CB = TG_THREADS / K;
  extern __shared__ __align__(16) unsigned char smraw[];
  R* mt = reinterpret_cast<R*>(smraw);     // [K][K] tmtx^T (l, k)
  R* mw = mt + K * K;                      // [K][K] ww^T (l, k)
  R* sw = mw + K * K;                      // [CB][K] div + padv
  R* sp = sw + CB * K;                     // [CB][K] padv
  R* sdv = sp + CB * K;                    // [CB][K] div
  R* sx = sdv + CB * K;                    // [CB][K] tv' - t
  R* s0s = sx + CB * K;                    // [CB] S[0]
  const size_t ncol2 = (size_t)J * I;
  const int tid = threadIdx.x, c = tid / K, k = tid - c * K;
  const size_t col = (size_t)blockIdx.x * CB + c;
  const bool act = c < CB && col < (size_t)a.nmem * ncol2;
  auto P = [](const void* p) { return (const R*)p; };
  for (int x = tid; x < K * K; x += TG_THREADS) {
    const int kk = x / K, l = x - kk * K;
    mt[l * K + kk] = P(a.tmtx)[x];
    mw[l * K + kk] = P(a.ww)[x];
  }
  const size_t e = act ? col / ncol2 : 0, ji = act ? col - e * ncol2 : 0;
  const R kappa = R(a.kappa), eps = R(a.epsvt), rair = R(a.rair);
  const R *dsig = P(a.dsig), *sigm = P(a.sigm);
  const size_t b3 = ji * K;                // basic-state column offset
  const size_t p3 = (act ? col : 0) * K;   // perturbation column offset
  const R *ub = P(a.ub) + b3, *vb = P(a.vb) + b3, *tb = P(a.tb) + b3, *qb = P(a.qb) + b3,
          *tvb = P(a.tvb) + b3, *absv = P(a.absvor) + b3, *divb = P(a.divb) + b3,
          *x5b = P(a.x5b) + b3, *sdb = P(a.sdotb) + ji * (K + 1);
  const R *u = P(a.u) + p3, *v = P(a.v) + p3, *t = P(a.t) + p3, *q = P(a.q) + p3,
          *vor = P(a.vor) + p3, *div = P(a.div) + p3;
  R pixb = R(0), piyb = R(0), pix = R(0), piy = R(0), padv = R(0), tv = R(0), dv = R(0);
  if (act) {
    pixb = P(a.pixb)[ji];
    piyb = P(a.piyb)[ji];
    pix = P(a.pix)[col];
    piy = P(a.piy)[col];
    dv = div[k];
    padv = u[k] * pixb + ub[k] * pix + v[k] * piyb + vb[k] * piy;
    tv = t[k] + eps * (t[k] * qb[k] + tb[k] * q[k]);     // tv'
    sw[tid] = dv + padv;
    sp[tid] = padv;
    sdv[tid] = dv;
    sx[tid] = tv - t[k];
  }
  __syncthreads();
  // S_k = sum_{l>=k} dsig_l (div + padv)_l  (dynamics.py:96-102)
  const int cK = c * K;
  R Sk1 = R(0), Sk = R(0);
  if (act) {
    for (int l = K - 1; l > k; --l) Sk1 = Sk1 + sw[cK + l] * dsig[l];
    Sk = Sk1 + sw[tid] * dsig[k];
    if (k == 0) s0s[c] = Sk;
    if (k == K - 1) {
      // gt_pi = -S[0] + sum dsig div (dynamics.py:188) = -sum dsig padv: summed
      // directly, without the cancellation of two O(div) terms
      R gtpi = R(0);
      for (int l = 0; l < K; ++l) gtpi -= sp[cK + l] * dsig[l];
      if (a.frc_ps) gtpi += P(a.frc_ps)[e * a.frc_ps_stride + ji];
      ((R*)a.gt_pi)[col] = gtpi;
    }
  }
  __syncthreads();
  if (!act) return;
  const R S0 = s0s[c];
  // sigma-dot at the half levels k and k + 1 (dynamics.py:105-114)
  const R sd0 = k == 0 ? R(0) : sigm[k] * S0 - Sk;
  const R sd1 = k == K - 1 ? R(0) : sigm[k + 1] * S0 - Sk1;
  const R sb0 = sdb[k], sb1 = sdb[k + 1], dsk = dsig[k], rdsk = R(1) / dsk;
  auto vadv = [&](const R* f, const R* fb) {
    return vert_adv<R>(k, K, [&](int l) { return f[l]; }, sb0, sb1, dsk, rdsk) +
           vert_adv<R>(k, K, [&](int l) { return fb[l]; }, sd0, sd1, dsk, rdsk);
  };
  const R x5p = P(a.alpha)[k] * dv + P(a.wP)[k] * padv + P(a.w3)[k] * Sk1;
  const R adiab = -kappa * (tv * x5b[k] + tvb[k] * x5p);
  const R tdev = tb[k] - P(a.tref)[k];
  ((R*)a.xu)[p3 + k] = u[k] * tdev + ub[k] * t[k];
  ((R*)a.xv)[p3 + k] = v[k] * tdev + vb[k] * t[k];
  const R hadv = t[k] * divb[k] + tdev * dv;
  R tm = R(0), phiv = R(0);
#pragma unroll 4
  for (int l = 0; l < K; ++l) {
    tm += sdv[cK + l] * mt[l * K + k];
    phiv += sx[cK + l] * mw[l * K + k];
  }
  R gtk = adiab + hadv + vadv(t, tb) + tm;
  if (a.frc_t) gtk += P(a.frc_t)[e * a.frc_t_stride + b3 + k];
  ((R*)a.gt)[p3 + k] = gtk;
  // momentum (dynamics.py:224-237)
  const R rcpg = rair * P(a.cpg)[k];
  const R tvdev = tvb[k] - P(a.tref)[k];
  R fuk = v[k] * absv[k] + vb[k] * vor[k];
  R fvk = -u[k] * absv[k] - ub[k] * vor[k];
  fuk -= rcpg * (tv * pixb + tvdev * pix);
  fvk -= rcpg * (tv * piyb + tvdev * piy);
  fuk += vadv(u, ub);
  fvk += vadv(v, vb);
  ((R*)a.fu)[p3 + k] = fuk;
  ((R*)a.fv)[p3 + k] = fvk;
  R kek = phiv + u[k] * ub[k] + v[k] * vb[k];
  if (a.lin_u)   // tangent-linear: linearised about the trajectory (lin_u, lin_v)
    kek += P(a.lin_u)[p3 + k] * u[k] + P(a.lin_v)[p3 + k] * v[k];
  else if (!a.strictly_linear)
    kek += R(0.5) * (u[k] * u[k] + v[k] * v[k]);
  ((R*)a.ke)[p3 + k] = kek;
  // humidity (dynamics.py:256-262)
  ((R*)a.yu)[p3 + k] = u[k] * qb[k] + ub[k] * q[k];
  ((R*)a.yv)[p3 + k] = v[k] * qb[k] + vb[k] * q[k];
  R gk = q[k] * divb[k] + qb[k] * dv + vert_adv<R>(k, K, [&](int l) { return q[l]; }, sb0, sb1, dsk, rdsk) +
         vert_adv<R>(k, K, [&](int l) { return qb[l]; }, sd0, sd1, dsk, rdsk);
  if (a.frc_q) gk += P(a.frc_q)[e * a.frc_q_stride + b3 + k];
  ((R*)a.g)[p3 + k] = gk;
  if (a.omega)
    ((R*)a.omega)[p3 + k] = -P(a.sig)[k] * (x5p * P(a.psb)[ji] + x5b[k] * P(a.ps)[col]);
  if (a.sdot) {
    R* o = (R*)a.sdot + col * (K + 1) + k;
    o[0] = sd0;
    if (k == K - 1) o[1] = sd1;
  }
}

// One block per (e, m, n) coefficient, thread per level.
template <typename R>
__global__ void k_implicit_rect(lbm_implicit_args a) {
  const int K = a.kmax, M = a.nmax + 1;
  const int n = blockIdx.x, m = blockIdx.y, e = blockIdx.z, k = threadIdx.x;
  __shared__ C2<R> sx[KMAX_LOCAL], sy[KMAX_LOCAL];
  const size_t o3 = (((size_t)e * M + m) * M + n) * K + k;
  const size_t o2 = ((size_t)e * M + m) * M + n;
  auto P = [](const void* p) { return (const R*)p; };
  C2<R>* nv = (C2<R>*)a.n_vor;
  C2<R>* nd = (C2<R>*)a.n_div;
  C2<R>* nt = (C2<R>*)a.n_t;
  C2<R>* nq = (C2<R>*)a.n_q;
  C2<R>* np = (C2<R>*)a.n_pi;
  const C2<R> z = cmk<R>(0, 0);
  if (n < m) {                      // outside the triangle: keep zeros
    if (k < K) { nv[o3] = z; nd[o3] = z; nt[o3] = z; nq[o3] = z; }
    if (k == 0) np[o2] = z;
    return;
  }
  const R dt = R(a.dt), dt2 = R(2) * dt;
  const R ktt = P(a.ktt)[n * K + k], kd = P(a.kd)[n * K + k];
  const R kv = P(a.kv)[n * K + k], kq = P(a.kq)[n * K + k];
  const R ft = R(1) + dt2 * ktt;
  const R lap = P(a.lap)[n];
  const C2<R> pt = ((const C2<R>*)a.p_t)[o3], wtt = ((const C2<R>*)a.w_t)[o3];
  // wdx = T(t-dt)(1 + dt ktt) + dt wt_t ; wdphix = WW wdx  (integrator.py:287-288)
  sx[k] = pt * (R(1) + dt * ktt) + wtt * dt;
  __syncthreads();
  C2<R> wdphix = z;
  for (int l = 0; l < K; ++l) cfma(wdphix, P(a.ww)[k * K + l], sx[l]);
  const C2<R> ppi = ((const C2<R>*)a.p_pi)[o2], wpi = ((const C2<R>*)a.w_pi)[o2];
  const C2<R> wdpix = ppi + wpi * dt;
  const C2<R> wdphiy = wdphix + wdpix * (ft * P(a.gg)[k]);
  const C2<R> pdv = ((const C2<R>*)a.p_div)[o3], wdv = ((const C2<R>*)a.w_div)[o3];
  const C2<R> rhs = pdv * ((R(1) + dt * kd) * ft) + (wdv * ft - wdphiy * lap) * dt;
  __syncthreads();
  sy[k] = rhs;
  __syncthreads();
  C2<R> dbar = z;
  const R* mi = P(a.minv) + (size_t)n * K * K;
  for (int l = 0; l < K; ++l) cfma(dbar, mi[k * K + l], sy[l]);
  __syncthreads();
  sx[k] = dbar;
  __syncthreads();
  C2<R> corr = z, dsum = z;
  for (int l = 0; l < K; ++l) {
    cfma(corr, P(a.tmtx)[k * K + l], sx[l]);
    cfma(dsum, P(a.dsig)[l], sx[l]);
  }
  const C2<R> wt2 = wtt - corr;
  const C2<R> wpi2 = wpi - dsum;
  const C2<R> pv = ((const C2<R>*)a.p_vor)[o3], wv = ((const C2<R>*)a.w_vor)[o3];
  const C2<R> pq = ((const C2<R>*)a.p_q)[o3], wq = ((const C2<R>*)a.w_q)[o3];
  C2<R> v_new = (pv + wv * dt2) * (R(1) / (R(1) + dt2 * kv));
  C2<R> d_new = dbar * R(2) - pdv;
  C2<R> t_new = (pt + wt2 * dt2) * (R(1) / ft);
  C2<R> q_new = (pq + wq * dt2) * (R(1) / (R(1) + dt2 * kq));
  if (k == 0) np[o2] = ppi + wpi2 * dt2;
  // implicit vertical diffusion (integrator.py:311-314), n = 0, 1 skipped for vor/div
  const void* vd[4] = {a.vd_vor, a.vd_div, a.vd_t, a.vd_q};
  C2<R>* vals[4] = {&v_new, &d_new, &t_new, &q_new};
  for (int f = 0; f < 4; ++f) {
    if (!vd[f]) continue;
    if (f < 2 && n < 2) continue;
    __syncthreads();
    sx[k] = *vals[f];
    __syncthreads();
    C2<R> o = z;
    for (int l = 0; l < K; ++l) cfma(o, P(vd[f])[k * K + l], sx[l]);
    *vals[f] = o;
  }
  nv[o3] = v_new;
  nd[o3] = d_new;
  nt[o3] = t_new;
  nq[o3] = q_new;
}

}  // namespace lbm

using namespace lbm;

extern "C" {

int lbm_tendency_grid(int prec, const lbm_tend_grid_args* a, void* stream) {
  if (!a || a->nmem < 1 || a->kmax < 1 || a->kmax > KMAX_LOCAL || a->nlat < 2 || a->nlon < 2)
    return LBM_ERR_ARG;
  if ((a->lin_u == nullptr) != (a->lin_v == nullptr)) return LBM_ERR_ARG;
  const size_t cols = (size_t)a->nmem * a->nlat * a->nlon;
  const int CB = TG_THREADS / a->kmax;
  const unsigned blocks = (unsigned)((cols + CB - 1) / CB);
  auto go = [&](auto kern, size_t smem) {
    if (smem > 48 * 1024) allow_smem(kern);   // (any kernel may have 48 KB)
    kern<<<blocks, TG_THREADS, smem, (cudaStream_t)stream>>>(*a);
  };
  if (prec == LBM_F64)
    go(k_tendency_grid<double>, tend_smem<double>(a->kmax));
  else if (prec == LBM_F32)
    go(k_tendency_grid<float>, tend_smem<float>(a->kmax));
  else
    return LBM_ERR_ARG;
  LBM_LAUNCH_CHECK();
  return LBM_OK;
}

int lbm_implicit_step(int prec, const lbm_implicit_args* a, void* stream) {
  if (!a || a->nmem < 1 || a->kmax < 1 || a->kmax > KMAX_LOCAL || a->nmax < 1) return LBM_ERR_ARG;
  const int M = a->nmax + 1;
  dim3 grid(M, M, a->nmem);
  if (prec == LBM_F64)
    k_implicit_rect<double><<<grid, a->kmax, 0, (cudaStream_t)stream>>>(*a);
  else if (prec == LBM_F32)
    k_implicit_rect<float><<<grid, a->kmax, 0, (cudaStream_t)stream>>>(*a);
  else
    return LBM_ERR_ARG;
  LBM_LAUNCH_CHECK();
  return LBM_OK;
}

}  // extern "C"
