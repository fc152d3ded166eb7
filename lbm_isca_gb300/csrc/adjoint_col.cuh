// Adjoints of the two per-column / per-coefficient linear maps of the time
// step, written once for the device kernels (adjoint.cu) and for host
// compilation (the CPU tests build this header with g++ and check it
// against the forward formulas).  Plain real arithmetic, no CUDA types.
//
// Forward maps (reference dynamics.py:156-271 and integrator.py:264-315):
//  * grid-point tendency, one column: inputs u v t q vor div [K] and pi_x
//    pi_y; outputs fu fv ke gt xu xv g yu yv [K] and gt_pi.  Linear about
//    the basic state except the kinetic energy 0.5 (u^2 + v^2), which is
//    linearised about a trajectory (u0, v0): ke += u0 u + v0 v.
//  * semi-implicit leapfrog update, one (m, n) coefficient: linear in the
//    previous level and the explicit tendencies, real coefficients, so the
//    real and imaginary parts go through the same transpose.
#pragma once

#if defined(__CUDACC__)
#define LBM_COL_HD __host__ __device__ inline
#else
#define LBM_COL_HD inline
#endif

namespace lbm_adj {

// Transposes of the vertical advection operator at one level,
//   VA(f; s)[k] = (fhi - flo - f[k] (s[k+1] - s[k])) / dsig[k],
//   flo = s[k] (f[k] + f[k-1]) / 2 for k >= 1, fhi = s[k+1] (f[k+1] + f[k]) / 2
//   for k + 1 <= K - 1 (reference dynamics.py:117-143), z = y / dsig.
// Of the f-argument: level k of fbar = dVA/df^T y, from z at k - 1, k, k + 1.
template <typename R>
LBM_COL_HD R va_f_adj(int k, int K, R zm, R z, R zp, R s0, R s1) {
  const R lo = k >= 1 ? R(0.5) * s0 * (zm - z) : R(0);
  const R hi = k + 1 <= K - 1 ? R(0.5) * s1 * (z - zp) : R(0);
  return lo + hi - z * (s1 - s0);
}

// Of the s-argument: half level k (1 <= k <= K - 1) of sbar = dVA/ds^T y.
template <typename R>
LBM_COL_HD R va_s_adj(R f, R fm, R z, R zm) { return R(0.5) * (f - fm) * (z + zm); }

// Vertical constants and one column of the basic state.
template <typename R>
struct ColConst {
  int K;
  R kappa, eps, rair;
  const R *dsig, *sigm, *alpha, *w3, *wP, *cpg, *ww, *tmtx, *tref;    // [K] / [K+1] / [K][K]
  const R *ub, *vb, *tb, *qb, *tvb, *absv, *divb, *x5b, *sdb;         // [K], sdb [K+1]
  R pixb, piyb;
  const R *u0, *v0;   // linearisation trajectory of the kinetic energy, or null
};

// Adjoints of the outputs of one column (each [K]; gt_pi: one value).
template <typename R>
struct TendAdjIn {
  const R *fu, *fv, *ke, *gt, *xu, *xv, *g, *yu, *yv;
  R gtpi;
};

// Level k of the adjoint of sigma-dot and of the column sums: sd'[k] =
// sigm[k] S[0] - S[k] for 1 <= k <= K-1 (zero at both ends), x5'[k-1] takes w3
// S[k].  sa: the adjoint of S[k], k >= 1; sb: this level's part of that of S[0].
template <typename R>
LBM_COL_HD void tendency_adj_sums(const ColConst<R>& c, const TendAdjIn<R>& y, int k, R* sa,
                                  R* sb) {
  *sa = *sb = R(0);
  if (k == 0) return;
  const R r = R(1) / c.dsig[k], rm = R(1) / c.dsig[k - 1];
  const R asd = va_s_adj(c.tb[k], c.tb[k - 1], y.gt[k] * r, y.gt[k - 1] * rm) +
                va_s_adj(c.ub[k], c.ub[k - 1], y.fu[k] * r, y.fu[k - 1] * rm) +
                va_s_adj(c.vb[k], c.vb[k - 1], y.fv[k] * r, y.fv[k - 1] * rm) +
                va_s_adj(c.qb[k], c.qb[k - 1], y.g[k] * r, y.g[k - 1] * rm);
  *sa = -c.w3[k - 1] * c.kappa * c.tvb[k - 1] * y.gt[k - 1] - asd;
  *sb = c.sigm[k] * asd;
}

// Adjoints of the inputs at level k: u v t q vor div and the level's parts of
// those of pi_x, pi_y.
template <typename R>
struct TendAdjOut { R u, v, t, q, vor, div, px, py; };

// cum: sum of the adjoints of S[0] .. S[k] (S[k] = sum_{l >= k} dsig_l (div' +
// padv')_l); gt, ke: the column's values again, in fast memory.
template <typename R>
LBM_COL_HD TendAdjOut<R> tendency_adj_level(const ColConst<R>& c, const TendAdjIn<R>& y, int k,
                                            R cum, const R* gt, const R* ke) {
  const int K = c.K;
  TendAdjOut<R> o;
  const R tdev = c.tb[k] - c.tref[k], tvdev = c.tvb[k] - c.tref[k];
  const R rcpg = c.rair * c.cpg[k];
  const R g = gt[k], fu = y.fu[k], fv = y.fv[k], e = ke[k], ag = y.g[k];
  const R s0 = c.sdb[k], s1 = c.sdb[k + 1];
  const R r = R(1) / c.dsig[k], rm = k >= 1 ? R(1) / c.dsig[k - 1] : R(0),
          rp = k + 1 <= K - 1 ? R(1) / c.dsig[k + 1] : R(0);
  const int km = k >= 1 ? k - 1 : 0, kp = k + 1 <= K - 1 ? k + 1 : k;
  auto vaf = [&](const R* a) {
    return va_f_adj(k, K, a[km] * rm, a[k] * r, a[kp] * rp, s0, s1);
  };
  // gt: + sum_l tmtx[k][l] div'_l;  ke: sum_l ww[k][l] (tv'_l - t'_l)
  R tm = R(0), he = R(0);
  for (int l = 0; l < K; ++l) {
    tm += c.tmtx[l * K + k] * gt[l];
    he += c.ww[l * K + k] * ke[l];
  }
  // gt = -kappa (tv' x5b + tvb x5') + t' divb + tdev div' + VA(t'; sdb) + VA(tb; sd')
  // fu = v' absv + vb vor' - rcpg (tv' pixb + tvdev pi_x) + VA(u'; sdb) + VA(ub; sd')
  // fv = -u' absv - ub vor' - rcpg (tv' piyb + tvdev pi_y) + VA(v'; sdb) + VA(vb; sd')
  const R atv = he - c.kappa * c.x5b[k] * g - rcpg * (c.pixb * fu + c.piyb * fv);
  const R ax5 = -c.kappa * c.tvb[k] * g;
  // x5' = alpha div' + wP padv' + w3 S[k+1];  gt_pi = -sum_k dsig padv'
  o.div = tdev * g + tm + c.qb[k] * ag + c.alpha[k] * ax5 + c.dsig[k] * cum;
  const R apadv = c.wP[k] * ax5 + c.dsig[k] * (cum - y.gtpi);
  // tv' = t' (1 + eps qb) + eps tb q';  xu = u' tdev + ub t', xv = v' tdev + vb t'
  o.t = c.divb[k] * g + vaf(y.gt) + c.ub[k] * y.xu[k] + c.vb[k] * y.xv[k] - he +
        (R(1) + c.eps * c.qb[k]) * atv;
  // g = q' divb + qb div' + VA(q'; sdb) + VA(qb; sd');  yu = u' qb + ub q', yv = v' qb + vb q'
  o.q = c.ub[k] * y.yu[k] + c.vb[k] * y.yv[k] + c.divb[k] * ag + vaf(y.g) +
        c.eps * c.tb[k] * atv;
  // ke: u' (ub + u0) + v' (vb + v0);  padv' = u' pixb + ub pi_x + v' piyb + vb pi_y
  o.u = tdev * y.xu[k] + vaf(y.fu) - c.absv[k] * fv + (c.ub[k] + (c.u0 ? c.u0[k] : R(0))) * e +
        c.qb[k] * y.yu[k] + c.pixb * apadv;
  o.v = tdev * y.xv[k] + vaf(y.fv) + c.absv[k] * fu + (c.vb[k] + (c.v0 ? c.v0[k] : R(0))) * e +
        c.qb[k] * y.yv[k] + c.piyb * apadv;
  o.vor = c.vb[k] * fu - c.ub[k] * fv;
  o.px = c.ub[k] * apadv - rcpg * tvdev * fu;
  o.py = c.vb[k] * apadv - rcpg * tvdev * fv;
  return o;
}

// Adjoint of the grid-point tendency of one column, level after level.  Inputs:
// adjoints of fu fv ke gt xu xv g yu yv (each [K]) and of gt_pi.  Outputs
// (overwritten): adjoints of u v t q vor div ([K]) and of pi_x, pi_y.  Scratch:
// 5 (K + 1) values in `work`.
template <typename R>
LBM_COL_HD void tendency_column_adjoint(const ColConst<R>& c, const R* afu, const R* afv,
                                        const R* ake, const R* agt, const R* axu,
                                        const R* axv, const R* ag, const R* ayu,
                                        const R* ayv, R agtpi, R* au, R* av, R* at, R* aq,
                                        R* avor, R* adiv, R* apix, R* apiy, R* work) {
  const TendAdjIn<R> y = {afu, afv, ake, agt, axu, axv, ag, ayu, ayv, agtpi};
  R cum = R(0), sb;
  for (int k = 0; k < c.K; ++k) {
    tendency_adj_sums(c, y, k, work + k, &sb);
    cum += sb;
  }
  *apix = *apiy = R(0);
  for (int k = 0; k < c.K; ++k) {
    cum += work[k];
    const TendAdjOut<R> o = tendency_adj_level(c, y, k, cum, agt, ake);
    au[k] = o.u;
    av[k] = o.v;
    at[k] = o.t;
    aq[k] = o.q;
    avor[k] = o.vor;
    adiv[k] = o.div;
    *apix += o.px;
    *apiy += o.py;
  }
}

// Operators of the implicit update for one total wavenumber n.
template <typename R>
struct ImplConst {
  int K;
  R dt, lap;                                  // time step, -n(n+1)/a^2
  const R *kv, *kd, *ktt, *kq;                // [K] at this n
  const R *ww, *tmtx, *gg, *dsig, *minv;      // [K][K], [K][K], [K], [K], [K][K] at this n
  const R* vd[4];                             // vertical diffusion of vor div t q, or null
  bool vd_skip_vordiv;                        // n < 2: no vertical diffusion of vor, div
};

// Element l of A^T x, for real or complex x.
template <typename R, typename V>
LBM_COL_HD V mat_t(const R* A, const V* x, int l, int K, V acc) {
  for (int k = 0; k < K; ++k) acc = acc + x[k] * A[k * K + l];
  return acc;
}

// Adjoint of the implicit update of one coefficient at level l, in four parts with
// the column's values of the part before between them (V: real, or complex).
template <typename V>
struct ImplAdjLevel { V ap[4], aw[4], x; };   // vor div t q of the previous level, of the
                                              // tendencies; the value the next part needs

// x = VD^T an (no diffusion of vor, div at n < 2), field f.
template <typename R, typename V>
LBM_COL_HD V impl_adj_vdiff(const ImplConst<R>& c, int f, const V* an, int l, V zero) {
  const bool use = c.vd[f] && !(f < 2 && c.vd_skip_vordiv);
  return use ? mat_t(c.vd[f], an, l, c.K, zero) : an[l];
}

// The pointwise updates: vor/q_new = (p + 2 dt w) / (1 + 2 dt kv|kq), d_new = 2 dbar - p_div,
// t_new = (p_t + 2 dt (w_t - tmtx dbar)) / ft.  Leaves the adjoint of dbar in x.
template <typename R, typename V>
LBM_COL_HD void impl_adj_point(const ImplConst<R>& c, int l, const V* v, ImplAdjLevel<V>& o) {
  const R dt2 = R(2) * c.dt;
  const R rv = R(1) / (R(1) + dt2 * c.kv[l]), rq = R(1) / (R(1) + dt2 * c.kq[l]);
  const R rt = R(1) / (R(1) + dt2 * c.ktt[l]);
  o.ap[0] = v[0] * rv;
  o.aw[0] = v[0] * (dt2 * rv);
  o.ap[1] = v[1] * R(-1);
  o.ap[2] = v[2] * rt;
  o.aw[2] = v[2] * (dt2 * rt);
  o.ap[3] = v[3] * rq;
  o.aw[3] = v[3] * (dt2 * rq);
  o.x = v[1] * R(2);
}

// pi_new = p_pi + 2 dt (w_pi - sum dsig dbar); awt: the aw[2] of the column.
template <typename R, typename V>
LBM_COL_HD void impl_adj_dbar(const ImplConst<R>& c, int l, const V* awt, V awpi, V zero,
                              ImplAdjLevel<V>& o) {
  o.x = o.x + mat_t(c.tmtx, awt, l, c.K, zero) * R(-1) + awpi * (-c.dsig[l]);
}

// dbar = Minv rhs, rhs = p_div (1 + dt kd) ft + dt (w_div ft - lap wdphiy), wdphiy =
// WW wdx + gg ft (p_pi + dt w_pi).  Leaves the adjoint of wdphiy in x; returns
// this level's part of that of p_pi.
template <typename R, typename V>
LBM_COL_HD V impl_adj_rhs(const ImplConst<R>& c, int l, const V* dbar, V zero,
                          ImplAdjLevel<V>& o) {
  const R ft = R(1) + R(2) * c.dt * c.ktt[l];
  const V rhs = mat_t(c.minv, dbar, l, c.K, zero);
  o.ap[1] = o.ap[1] + rhs * ((R(1) + c.dt * c.kd[l]) * ft);
  o.aw[1] = rhs * (c.dt * ft);
  o.x = rhs * (-c.dt * c.lap);
  return o.x * (c.gg[l] * ft);
}

// wdx = p_t (1 + dt ktt) + dt w_t
template <typename R, typename V>
LBM_COL_HD void impl_adj_wdx(const ImplConst<R>& c, int l, const V* phy, V zero,
                             ImplAdjLevel<V>& o) {
  const V s = mat_t(c.ww, phy, l, c.K, zero);
  o.ap[2] = o.ap[2] + s * (R(1) + c.dt * c.ktt[l]);
  o.aw[2] = o.aw[2] + s * c.dt;
}

// The four parts for one coefficient and one real component (stride `st`
// between levels).  Inputs: adjoints of the new level an_* [K] and an_pi.
// Outputs (overwritten): adjoints of the previous level ap_* and of the explicit
// tendencies aw_*.  Scratch: 4 K values.
template <typename R>
LBM_COL_HD void implicit_coef_adjoint(const ImplConst<R>& c, int st, const R* an_vor,
                                      const R* an_div, const R* an_t, const R* an_q, R an_pi,
                                      R* ap_vor, R* ap_div, R* ap_t, R* ap_q, R* ap_pi,
                                      R* aw_vor, R* aw_div, R* aw_t, R* aw_q, R* aw_pi,
                                      R* work) {
  const int K = c.K;
  const R* an[4] = {an_vor, an_div, an_t, an_q};
  R* ap[4] = {ap_vor, ap_div, ap_t, ap_q};
  R* aw[4] = {aw_vor, aw_div, aw_t, aw_q};
  R *col = work, *x = work + K, *y = work + 2 * K, *cp = work + 3 * K;
  auto get = [&](int l) {
    ImplAdjLevel<R> o;
    for (int f = 0; f < 4; ++f) { o.ap[f] = ap[f][l * st]; o.aw[f] = aw[f][l * st]; }
    o.x = x[l];
    return o;
  };
  auto put = [&](int l, const ImplAdjLevel<R>& o, R* next) {
    for (int f = 0; f < 4; ++f) { ap[f][l * st] = o.ap[f]; aw[f][l * st] = o.aw[f]; }
    next[l] = o.x;
  };
  for (int f = 0; f < 4; ++f) {
    for (int k = 0; k < K; ++k) cp[k] = an[f][k * st];
    for (int l = 0; l < K; ++l) ap[f][l * st] = impl_adj_vdiff(c, f, cp, l, R(0));
  }
  for (int l = 0; l < K; ++l) {
    ImplAdjLevel<R> o = {};
    const R v[4] = {ap[0][l * st], ap[1][l * st], ap[2][l * st], ap[3][l * st]};
    impl_adj_point(c, l, v, o);
    put(l, o, x);
    col[l] = o.aw[2];
  }
  *ap_pi = an_pi;
  *aw_pi = R(2) * c.dt * an_pi;
  for (int l = 0; l < K; ++l) {
    ImplAdjLevel<R> o = get(l);
    impl_adj_dbar(c, l, col, *aw_pi, R(0), o);
    put(l, o, y);
  }
  R apix = R(0);
  for (int l = 0; l < K; ++l) {
    ImplAdjLevel<R> o = get(l);
    apix += impl_adj_rhs(c, l, y, R(0), o);
    put(l, o, x);
  }
  *ap_pi += apix;
  *aw_pi += c.dt * apix;
  for (int l = 0; l < K; ++l) {
    ImplAdjLevel<R> o = get(l);
    impl_adj_wdx(c, l, x, R(0), o);
    put(l, o, y);
  }
}

}  // namespace lbm_adj
