// Fused ensemble stepper: the per-step hot path of LBM.run
// (model.py:213-247) for many members at once, with the prognostic state in
// packed spectral space.
//
// One step = four parts (each one launch or more):
//   grid part   three launches (k_ifft / k_idft, k_alg, k_ffft / k_fdft:
//               grid_split.cuh, grid_fft.cuh) where the caller gives buffers
//               for the grid rows (always in FP32), else
//   k_grid      per (member, latitude): inverse FFTs of the synthesised
//               Fourier fields, the whole grid-point tendency algebra of
//               dynamics.py:176-262 level by level, forward FFTs, weighting;
//               also the grid-space Robert-Asselin filter of ps (state.py
//               :110-128 acts on ps, which is nonlinear in pi).
//   k_anal      per (member, m-pair, level chunk): Legendre analysis with the
//               equatorial symmetry split -> explicit spectral tendencies.
//   k_implicit  per (member, n-pair): semi-implicit solve, leapfrog, implicit
//               damping / vertical diffusion, spectral Robert-Asselin filter
//               (integrator.py:264-315, state.py:110-128), column sums.
//   k_synth     per (member, m-pair, level chunk): Legendre synthesis of the
//               new level -> Fourier fields for the next k_grid.
//
// The reference keeps its state in grid space; u, v, T, q are band-limited,
// so filtering and advancing them in spectral space is exact to round-off.
// ps is not band-limited after its filter, so its two grid levels are kept.
// The column sum of dsig*(div + v.grad ln ps) that defines sigma-dot is
// split into its linear parts, which are synthesised from sigma-weighted
// column sums of psi, chi and div computed in k_implicit; k_grid then needs
// no second pass over the levels.
#include "lbm_common.cuh"
#include "lbm_fft.cuh"
#include "async_copy.cuh"
#include "tc_common.cuh"
#include <cmath>
#include <mutex>
#include <new>
#include <type_traits>

namespace lbm {

// ---- typed view of the descriptor ---------------------------------------------
template <typename R> struct SD {
  int E, J, I, N, M, K, NS, nsets, strictly_linear, frc_shared;
  int vd_on[4];
  R kappa, epsvt, robert;
  const R *symp, *symh;
  const C2<R>* tw;
  const R *jfac, *vert, *b3, *bsd, *b2;
  const R *lap, *invlap, *nn1a, *kv, *kd, *ktt, *kq, *ww, *tmtx, *minv, *vdiff;
  const C2<R> *frc3, *frcs;
  const float2* dft;
  C2<R> *sa3, *sas, *sb3;
  R *psa, *psb;
  C2<R> *sf, *sfs, *af, *afs, *tend, *tends;
  R *grid6, *grid9;
  int* err;
  int* err_member;
  int legendre;                          // 0 FMA; 3 or 6: tensor-core products
  const unsigned char* tc_anal;          // table image of k_anal_tc
  const unsigned char* tc_synth;         // table image of k_synth_tc
  int tc_off;                            // bits 0 / 1 / 2: Legendre analysis / synthesis,
                                         // longitude analysis on FMA
  int tc_g;                              // members per MMA tile cap (0: as many as fit)
  const unsigned char* tc_dft;           // table image of k_fdft_tc
};

template <typename R> SD<R> make_sd(const lbm_stepper_desc& d) {
  SD<R> s;
  s.E = d.nmem; s.J = d.nlat; s.I = d.nlon; s.N = d.nmax; s.M = d.nmax + 1; s.K = d.kmax;
  s.NS = nspec(d.nmax); s.nsets = d.nsets; s.strictly_linear = d.strictly_linear;
  s.frc_shared = d.frc_shared;
  for (int i = 0; i < 4; ++i) s.vd_on[i] = d.vd_on[i];
  s.kappa = R(d.kappa); s.epsvt = R(d.epsvt); s.robert = R(d.robert);
  s.symp = (const R*)d.symp; s.symh = (const R*)d.symh; s.tw = (const C2<R>*)d.tw;
  s.jfac = (const R*)d.jfac; s.vert = (const R*)d.vert; s.b3 = (const R*)d.b3;
  s.bsd = (const R*)d.bsd; s.b2 = (const R*)d.b2;
  s.lap = (const R*)d.lap; s.invlap = (const R*)d.invlap; s.nn1a = (const R*)d.nn1a;
  s.kv = (const R*)d.kv; s.kd = (const R*)d.kd; s.ktt = (const R*)d.ktt; s.kq = (const R*)d.kq;
  s.ww = (const R*)d.ww; s.tmtx = (const R*)d.tmtx; s.minv = (const R*)d.minv;
  s.vdiff = (const R*)d.vdiff;
  s.frc3 = (const C2<R>*)d.frc3; s.frcs = (const C2<R>*)d.frcs;
  s.dft = (const float2*)d.dft;
  s.sa3 = (C2<R>*)d.sa3; s.sas = (C2<R>*)d.sas; s.sb3 = (C2<R>*)d.sb3;
  s.psa = (R*)d.psa; s.psb = (R*)d.psb;
  s.sf = (C2<R>*)d.sf; s.sfs = (C2<R>*)d.sfs; s.af = (C2<R>*)d.af; s.afs = (C2<R>*)d.afs;
  s.tend = (C2<R>*)d.tend; s.tends = (C2<R>*)d.tends;
  s.grid6 = (R*)d.grid6; s.grid9 = (R*)d.grid9;
  s.err = d.err;
  s.err_member = d.err_member;
  s.legendre = d.legendre;
  s.tc_anal = (const unsigned char*)d.tc_anal;
  s.tc_synth = (const unsigned char*)d.tc_synth;
  s.tc_off = d.tc_off;
  s.tc_g = d.tc_g;
  s.tc_dft = (const unsigned char*)d.tc_dft;
  return s;
}

// basic-state 3-D field indices in b3 [10][J][K][I]
enum { B_U = 0, B_V, B_T, B_Q, B_TV, B_ABSVOR, B_DIV, B_X5, B_TDEV, B_TVDEV,
       B_HDU, B_HDV, B_HDT, B_HDQ, B_N };
// b2 [5][J][I]
enum { B2_PIX = 0, B2_PIY, B2_PSBAR, B2_USUM, B2_VSUM };
// jfac [4][J]
enum { JF_GW = 0, JF_GWDELC, JF_RCOS, JF_COS };
// Fourier field slots
enum { SF_U = 0, SF_V, SF_VOR, SF_DIV, SF_T, SF_Q, SF_N };           // sf [..][6]
enum { SFS_PI = 0, SFS_PIY, SFS_UH, SFS_VH, SFS_DH, SFS_N };         // sfs [..][5]
enum { AF_FU = 0, AF_FV, AF_KE, AF_T, AF_XV, AF_Q, AF_YV, AF_N };     // af [..][7]

template <typename R> LBM_D R vrow(const SD<R>& d, int row, int k) {
  return d.vert[row * (d.K + 1) + k];
}

// =============================================================================
// k_grid: Fourier -> grid -> tendency algebra -> Fourier, per (member, lat)
// =============================================================================
template <typename R, int I, int KB, int NT> struct GridSmem {
  static constexpr int R1 = FftShape<I>::R1;
  static constexpr int NTEAM = NT / R1;
  static constexpr int SCR = fft_team_scratch<I>();
  static constexpr int RS = KB + 2;          // ring slots of grid levels
  static constexpr int NG = 9;               // grid outputs per level
  static constexpr int NIN = (KB + 1) * SF_N;   // Fourier staging in (levels)
  static constexpr int NOUT = KB * AF_N;         // Fourier staging out
  static size_t bytes(int M) {
    return sizeof(C2<R>) * (size_t)(I + NTEAM * SCR + (NIN + NOUT) * M) +
           sizeof(R) * (size_t)I * (RS * SF_N + KB * NG + KB * 5 + 8 + 3);
  }
};

template <typename R> LBM_D R vadv(R fm, R f0, R fp, R s0, R s1, bool lo, bool hi, R dsk) {
  const R flo = lo ? s0 * R(0.5) * (f0 + fm) : R(0);
  const R fhi = hi ? s1 * R(0.5) * (fp + f0) : R(0);
  return (fhi - flo - f0 * (s1 - s0)) / dsk;
}

template <typename R, int I, int KB, int NT>
__global__ void __launch_bounds__(NT) k_grid(SD<R> d, int ps_mode) {
  using SM = GridSmem<R, I, KB, NT>;
  constexpr int R1 = SM::R1, NTEAM = SM::NTEAM, SCR = SM::SCR, RS = SM::RS, NG = SM::NG;
  const int j = blockIdx.x, e = blockIdx.y;
  const int J = d.J, K = d.K, M = d.M;
  const int tid = threadIdx.x, team = tid / R1, t = tid % R1;
  extern __shared__ unsigned char smraw[];
  C2<R>* tw = reinterpret_cast<C2<R>*>(smraw);
  C2<R>* scr = tw + I;
  C2<R>* fin = scr + NTEAM * SCR;                     // [KB+1][6][M] (or [5][M])
  C2<R>* fout = fin + SM::NIN * M;                     // [KB][7][M] (or [2][M])
  R* gin = reinterpret_cast<R*>(fout + SM::NOUT * M);  // [RS][6][I]
  R* gout = gin + RS * SF_N * I;                       // [KB][9][I]
  R* pre = gout + KB * NG * I;                         // [KB][5][I]
  R* sg = pre + KB * 5 * I;                            // [8][I] surface fields
  R* pst = sg + 8 * I;                                 // [3][I] running column prefixes
  for (int c = tid; c < I; c += NT) pst[c] = pst[I + c] = pst[2 * I + c] = R(0);

  for (int p = tid; p < I; p += NT) tw[p] = d.tw[p];
  const R gw = d.jfac[JF_GW * J + j], gwdc = d.jfac[JF_GWDELC * J + j];
  const R rcos = d.jfac[JF_RCOS * J + j];
  const R invI = R(1) / R(I);
  const size_t jmK = (size_t)J * K;
  const C2<R>* sfe = d.sf + (size_t)e * M * jmK * SF_N;
  C2<R>* afe = d.af + (size_t)e * M * jmK * AF_N;

  // ---- surface pre-pass ----------------------------------------------------
  for (int idx = tid; idx < M * SFS_N; idx += NT) {
    const int m = idx / SFS_N, f = idx % SFS_N;
    fin[f * M + m] = d.sfs[(((size_t)e * M + m) * J + j) * SFS_N + f];
  }
  __syncthreads();
  // jobs: 0 pi, 1 pi_x (i m pi, /(a cos)), 2 pi_y, 3 U-sum, 4 V-sum, 5 D-sum
  for (int job = team; job < 6; job += NTEAM) {
    const int src = (job <= 1) ? SFS_PI : job - 1;   // PI, PI, PIY, UH, VH, DH
    const C2<R>* X = fin + src * M;
    const R sc = (job == 0 || job == 5) ? R(1) : rcos;
    if (job == 1)
      team_rfft_inv<I>(t, [&](int m) { return im_mul(X[m], R(m)); }, M, scr + team * SCR, tw,
                       sg + job * I, 1, sc);
    else
      team_rfft_inv<I>(t, [&](int m) { return X[m]; }, M, scr + team * SCR, tw, sg + job * I,
                       1, sc);
  }
  __syncthreads();
  // per column: total column sum S_tot, gt_pi, ps update, pi(t - dt)
  const R* b2 = d.b2;
  for (int c = tid; c < I; c += NT) {
    const size_t g2 = (size_t)j * I + c;
    const R pixb = b2[(B2_PIX * J) * I + g2], piyb = b2[(B2_PIY * J) * I + g2];
    const R psbar = b2[(B2_PSBAR * J) * I + g2];
    const R usum = b2[(B2_USUM * J) * I + g2], vsum = b2[(B2_VSUM * J) * I + g2];
    const R pi = sg[0 * I + c], pix = sg[1 * I + c], piy = sg[2 * I + c];
    const R uh = sg[3 * I + c], vh = sg[4 * I + c], dh = sg[5 * I + c];
    const R stot = dh + pixb * uh + piyb * vh + pix * usum + piy * vsum;
    sg[6 * I + c] = stot;
    sg[7 * I + c] = dh;
    gout[0 * I + c] = dh - stot;                 // gt_pi (dynamics.py:188)
    const size_t gp = (size_t)e * J * I + g2;
    const R pscur = psbar * expm1(pi);           // state.py:81-83
    R pb = d.psb[gp];
    if (ps_mode == 1) {
      pb = d.psa[gp];
    } else if (ps_mode == 2) {
      const R pa = d.psa[gp];
      pb = pa + d.robert * (pb - R(2) * pa + pscur);
    }
    if (ps_mode != 0) {
      d.psb[gp] = pb;
      d.psa[gp] = pscur;
    }
    gout[1 * I + c] = log1p(pb / psbar);         // pi' of the filtered t - dt level
  }
  __syncthreads();
  for (int job = team; job < 2; job += NTEAM) {
    C2<R>* Y = fout + job * M;
    team_rfft_fwd<I>(t, gout + job * I, 1, scr + team * SCR, tw, M, gw * invI,
                     [&](int m, C2<R> X) { Y[m] = X; });
  }
  __syncthreads();
  for (int idx = tid; idx < M * 2; idx += NT) {
    const int m = idx / 2, f = idx % 2;
    d.afs[(((size_t)e * M + m) * J + j) * 2 + f] = fout[f * M + m];
  }

  // ---- level loop -----------------------------------------------------------
  const R eps = d.epsvt, kappa = d.kappa;
  const R* b3 = d.b3;
  auto B3 = [&](int f, int k, int c) -> R { return b3[(((size_t)f * J + j) * K + k) * I + c]; };
  auto BSD = [&](int k, int c) -> R { return d.bsd[((size_t)j * (K + 1) + k) * I + c]; };
  auto GIN = [&](int k, int f) -> R* { return gin + ((k % RS) * SF_N + f) * I; };

  for (int k0 = 0; k0 < K; k0 += KB) {
    const int lo = (k0 == 0) ? 0 : k0 + 1;
    const int hi = min(k0 + KB, K - 1);
    const int nl = hi - lo + 1;                 // levels to load (may be 0)
    __syncthreads();
    if (nl > 0) {
      for (int idx = tid; idx < M * nl * SF_N; idx += NT) {
        const int m = idx / (nl * SF_N), r = idx % (nl * SF_N);
        const int l = r / SF_N, f = r % SF_N;
        fin[(l * SF_N + f) * M + m] = sfe[((size_t)m * J + j) * K * SF_N + (size_t)(lo + l) * SF_N + f];
      }
      __syncthreads();
      for (int job = team; job < nl * SF_N; job += NTEAM) {
        const int l = job / SF_N, f = job % SF_N;
        const C2<R>* X = fin + (l * SF_N + f) * M;
        const R sc = (f == SF_U || f == SF_V) ? rcos : R(1);
        team_rfft_inv<I>(t, [&](int m) { return X[m]; }, M, scr + team * SCR, tw,
                         GIN(lo + l, f), 1, sc);
      }
      __syncthreads();
    }
    const int kb = min(KB, K - k0);             // levels processed this iteration
    // column prefixes (one thread per column, levels in order)
    for (int c = tid; c < I; c += NT) {
      const size_t g2 = (size_t)j * I + c;
      const R pixb = b2[(B2_PIX * J) * I + g2], piyb = b2[(B2_PIY * J) * I + g2];
      const R pix = sg[1 * I + c], piy = sg[2 * I + c], stot = sg[6 * I + c],
              dh = sg[7 * I + c];
      R pref = pst[c], prefd = pst[I + c], pref3 = pst[2 * I + c];
      for (int l = 0; l < kb; ++l) {
        const int k = k0 + l;
        const R u = GIN(k, SF_U)[c], v = GIN(k, SF_V)[c], dv = GIN(k, SF_DIV)[c];
        const R tt = GIN(k, SF_T)[c], q = GIN(k, SF_Q)[c];
        const R padv = u * pixb + B3(B_U, k, c) * pix + v * piyb + B3(B_V, k, c) * piy;
        R* pr = pre + (l * 5) * I;
        pr[0 * I + c] = stot - pref;                       // S[k]
        pref += (dv + padv) * vrow(d, LBM_VERT_DSIG, k);
        pr[1 * I + c] = stot - pref;                       // S[k+1]
        prefd += dv * vrow(d, LBM_VERT_DSIG, k);
        pr[2 * I + c] = dh - prefd;                        // sum_{l>k} dsig div
        const R x = eps * (tt * B3(B_Q, k, c) + B3(B_T, k, c) * q);   // Tv' - T'
        pr[3 * I + c] = pref3 + vrow(d, LBM_VERT_RALPHA, k) * x;      // (WW x)_k
        pref3 += vrow(d, LBM_VERT_RDLOG3, k) * x;
        pr[4 * I + c] = padv;
      }
      pst[c] = pref;
      pst[I + c] = prefd;
      pst[2 * I + c] = pref3;
    }
    __syncthreads();
    // pointwise algebra, (level, column) per thread
    for (int it = tid; it < kb * I; it += NT) {
      const int l = it / I, c = it % I, k = k0 + l;
      const size_t g2 = (size_t)j * I + c;
      const R pixb = b2[(B2_PIX * J) * I + g2], piyb = b2[(B2_PIY * J) * I + g2];
      const R pix = sg[1 * I + c], piy = sg[2 * I + c], stot = sg[6 * I + c];
      const R* pr = pre + (l * 5) * I;
      const R S0 = pr[0 * I + c], S1 = pr[1 * I + c], sdv = pr[2 * I + c];
      const R phiv = pr[3 * I + c], padv = pr[4 * I + c];
      const bool hasm = k >= 1, hasp = k + 1 <= K - 1;
      const int km = hasm ? k - 1 : k, kp = hasp ? k + 1 : k;
      const R sd0 = hasm ? vrow(d, LBM_VERT_SIGM, k) * stot - S0 : R(0);
      const R sd1 = hasp ? vrow(d, LBM_VERT_SIGM, k + 1) * stot - S1 : R(0);
      const R sb0 = BSD(k, c), sb1 = BSD(k + 1, c);
      const R dsk = vrow(d, LBM_VERT_DSIG, k);
      const R u = GIN(k, SF_U)[c], v = GIN(k, SF_V)[c], vo = GIN(k, SF_VOR)[c];
      const R dv = GIN(k, SF_DIV)[c], tt = GIN(k, SF_T)[c], q = GIN(k, SF_Q)[c];
      const R ub = B3(B_U, k, c), vb = B3(B_V, k, c), tb = B3(B_T, k, c), qb = B3(B_Q, k, c);
      const R tvb = B3(B_TV, k, c), absv = B3(B_ABSVOR, k, c), divb = B3(B_DIV, k, c);
      const R x5b = B3(B_X5, k, c), tdev = B3(B_TDEV, k, c), tvdev = B3(B_TVDEV, k, c);
      const R tv = tt + eps * (tt * qb + tb * q);
      const R x5p = vrow(d, LBM_VERT_ALPHA, k) * dv + vrow(d, LBM_VERT_WP, k) * padv +
                    vrow(d, LBM_VERT_W3, k) * S1;
      const R adiab = -kappa * (tv * x5b + tvb * x5p);
      const R hadv = tt * divb + tdev * dv;
      const R vadvT = vadv(GIN(km, SF_T)[c], tt, GIN(kp, SF_T)[c], sb0, sb1, hasm, hasp, dsk) +
                      vadv(B3(B_T, km, c), tb, B3(B_T, kp, c), sd0, sd1, hasm, hasp, dsk);
      const R tm = vrow(d, LBM_VERT_KTREF, k) *
                   (vrow(d, LBM_VERT_ALPHA, k) * dv + vrow(d, LBM_VERT_W3, k) * sdv);
      R* go = gout + (l * NG) * I;
      go[3 * I + c] = adiab + hadv + vadvT + tm;                          // gt_t
      go[4 * I + c] = u * tdev + ub * tt;                                 // xu
      go[5 * I + c] = v * tdev + vb * tt;                                 // xv
      const R rcpg = vrow(d, LBM_VERT_RCPG, k);
      R fu = v * absv + vb * vo - rcpg * (tv * pixb + tvdev * pix);
      R fv = -u * absv - ub * vo - rcpg * (tv * piyb + tvdev * piy);
      fu += vadv(GIN(km, SF_U)[c], u, GIN(kp, SF_U)[c], sb0, sb1, hasm, hasp, dsk) +
            vadv(B3(B_U, km, c), ub, B3(B_U, kp, c), sd0, sd1, hasm, hasp, dsk);
      fv += vadv(GIN(km, SF_V)[c], v, GIN(kp, SF_V)[c], sb0, sb1, hasm, hasp, dsk) +
            vadv(B3(B_V, km, c), vb, B3(B_V, kp, c), sd0, sd1, hasm, hasp, dsk);
      go[0 * I + c] = fu;
      go[1 * I + c] = fv;
      R ke = phiv + u * ub + v * vb;
      if (!d.strictly_linear) ke += R(0.5) * (u * u + v * v);
      go[2 * I + c] = ke;
      go[6 * I + c] = q * divb + qb * dv +
                      vadv(GIN(km, SF_Q)[c], q, GIN(kp, SF_Q)[c], sb0, sb1, hasm, hasp, dsk) +
                      vadv(B3(B_Q, km, c), qb, B3(B_Q, kp, c), sd0, sd1, hasm, hasp, dsk);
      go[7 * I + c] = u * qb + ub * q;                                    // yu
      go[8 * I + c] = v * qb + vb * q;                                    // yv
    }
    __syncthreads();
    // forward FFTs, weighted and combined into the 7 analysis inputs
    const R wd = gwdc * invI, wg = gw * invI;
    for (int job = team; job < kb * AF_N; job += NTEAM) {
      const int l = job / AF_N, a = job % AF_N;
      const R* go = gout + (l * NG) * I;
      C2<R>* Y = fout + (l * AF_N + a) * M;
      C2<R>* sc_ = scr + team * SCR;
      switch (a) {
        case AF_FU: team_rfft_fwd<I>(t, go + 0 * I, 1, sc_, tw, M, wd, [&](int m, C2<R> X) { Y[m] = X; }); break;
        case AF_FV: team_rfft_fwd<I>(t, go + 1 * I, 1, sc_, tw, M, wd, [&](int m, C2<R> X) { Y[m] = X; }); break;
        case AF_KE: team_rfft_fwd<I>(t, go + 2 * I, 1, sc_, tw, M, wg, [&](int m, C2<R> X) { Y[m] = X; }); break;
        case AF_T:
          team_rfft_fwd<I>(t, go + 3 * I, 1, sc_, tw, M, wg, [&](int m, C2<R> X) { Y[m] = X; });
          team_rfft_fwd<I>(t, go + 4 * I, 1, sc_, tw, M, wd,
                           [&](int m, C2<R> X) { Y[m] = Y[m] - im_mul(X, R(m)); });
          break;
        case AF_XV: team_rfft_fwd<I>(t, go + 5 * I, 1, sc_, tw, M, wd, [&](int m, C2<R> X) { Y[m] = X; }); break;
        case AF_Q:
          team_rfft_fwd<I>(t, go + 6 * I, 1, sc_, tw, M, wg, [&](int m, C2<R> X) { Y[m] = X; });
          team_rfft_fwd<I>(t, go + 7 * I, 1, sc_, tw, M, wd,
                           [&](int m, C2<R> X) { Y[m] = Y[m] - im_mul(X, R(m)); });
          break;
        default: team_rfft_fwd<I>(t, go + 8 * I, 1, sc_, tw, M, wd, [&](int m, C2<R> X) { Y[m] = X; }); break;
      }
    }
    __syncthreads();
    for (int idx = tid; idx < M * kb * AF_N; idx += NT) {
      const int m = idx / (kb * AF_N), r = idx % (kb * AF_N);
      const int l = r / AF_N, a = r % AF_N;
      afe[((size_t)m * J + j) * K * AF_N + (size_t)(k0 + l) * AF_N + a] = fout[(l * AF_N + a) * M + m];
    }
  }
}

// column sums of a freshly loaded current level
template <typename R>
__global__ void k_colsum(SD<R> d) {
  const int e = blockIdx.y;
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  const int NS = d.NS, K = d.K;
  if (idx >= NS) return;
  int m = 0;
  while (m < d.N && spec_offset(m + 1, d.N) <= idx) ++m;
  const int n = m + (idx - spec_offset(m, d.N));
  const size_t e3 = (size_t)e * 4 * NS * K;
  C2<R> sv = cmk<R>(0, 0), sdv = cmk<R>(0, 0);
  for (int l = 0; l < K; ++l) {
    cfma(sv, vrow(d, LBM_VERT_DSIG, l), d.sa3[e3 + 0 * NS * K + (size_t)idx * K + l]);
    cfma(sdv, vrow(d, LBM_VERT_DSIG, l), d.sa3[e3 + 1 * NS * K + (size_t)idx * K + l]);
  }
  const R il = d.invlap[n];
  const size_t es = (size_t)e * 4 * NS;
  d.sas[es + 1 * NS + idx] = sv * il;
  d.sas[es + 2 * NS + idx] = sdv * il;
  d.sas[es + 3 * NS + idx] = sdv;
}

// Apply the pending grid-ps update at the end of a run (see k_grid).
template <typename R, int I>
__global__ void k_ps_flush(SD<R> d, int ps_mode) {
  constexpr int R1 = FftShape<I>::R1;
  constexpr int SCR = fft_team_scratch<I>();
  const int j = blockIdx.x, e = blockIdx.y, J = d.J, M = d.M;
  __shared__ C2<R> tw[I];
  __shared__ C2<R> scr[SCR];
  __shared__ C2<R> X[I / 2];
  __shared__ R pi[I];
  const int tid = threadIdx.x;
  for (int p = tid; p < I; p += R1) tw[p] = d.tw[p];
  for (int m = tid; m < M; m += R1) X[m] = d.sfs[(((size_t)e * M + m) * J + j) * SFS_N + SFS_PI];
  __syncwarp();
  team_rfft_inv<I>(tid, [&](int m) { return X[m]; }, M, scr, tw, pi, 1, R(1));
  __syncwarp();
  for (int c = tid; c < I; c += R1) {
    const size_t g2 = (size_t)j * I + c;
    const size_t gp = (size_t)e * J * I + g2;
    const R psbar = d.b2[(B2_PSBAR * J) * I + g2];
    const R pscur = psbar * expm1(pi[c]);
    if (ps_mode == 1) {
      d.psb[gp] = d.psa[gp];
    } else if (ps_mode == 2) {
      const R pa = d.psa[gp];
      d.psb[gp] = pa + d.robert * (d.psb[gp] - R(2) * pa + pscur);
    }
    d.psa[gp] = pscur;
  }
}

}  // namespace lbm
#include "legendre_fma.cuh"
#include "implicit.cuh"
#include "grid_split.cuh"
#include "grid_fft.cuh"
#include "legendre_tc.cuh"
#include "synth_tc.cuh"
#include "dft_tc.cuh"
namespace lbm {

// ---- launch configuration ------------------------------------------------------
// Levels per segment of k_alg, 0 for whole columns: segments while the columns are
// less than a warp per SM partition (one member of T42: 256 of 608).  Two
// levels in FP32, bound by latency (T42L20, one member, us: 22 whole, 9.0, 10.6, 11.6
// and 17 with 2, 3, 5, 10 levels); five in FP64, where the sums below a segment
// cost more of the FP64 pipe (83 whole, 59, 50, 47, 52).  At 512 warps FP32 19.7 ->
// 15, FP64 84 either way; at 768 whole columns are as fast or faster (20.2 against
// 20.4, 106 against 140).
template <typename R> int alg_seg(int E, int J, int I, int K) {
  const long warps = (long)E * J * (I / 32);
  if (warps > 4 * FILL_SMS || K < 2) return 0;
  const int ls = sizeof(R) == 4 ? 2 : 5, least = (K + ALG_SEGMAX - 1) / ALG_SEGMAX;
  return ls > least ? ls : least;
}
template <int I> constexpr int alg_minb() { return I == 64 ? 10 : (I == 128 ? 6 : 3); }

template <typename R, int I> constexpr int grid_kb() { return (sizeof(R) == 8 && I == 256) ? 2 : 4; }
template <typename R, int I> constexpr int grid_nt() {
  return I == 64 ? 128 : ((I == 256 && sizeof(R) == 8) ? 128 : 256);
}

inline int persistent_grid(const void* fn, int nt, size_t smem, int units);
// Legendre synthesis launch; with the level fields on the tensor cores a second
// kernel makes the surface fields.
template <typename R> void launch_synth(const SD<R>& d, cudaStream_t st, bool attrs) {
  const SynthPlan sp = synth_plan<R>(d.E, d.J, d.K, d.N);
  const int NP = (d.M + 1) / 2;
  if constexpr (sizeof(R) == 4) {
    if (d.legendre && !(d.tc_off & 2)) {
      const StcPlan pl = stc_plan(d.E, d.J, d.K, d.N, d.tc_g);
      const int sm = sp.ox + (int)sizeof(C2<R>) * 4 * (d.N + 2);
      if (attrs) {
        allow_smem(k_synth_surf);
        return;
      }
      k_synth_tc<<<persistent_grid((const void*)k_synth_tc, STC_THREADS, pl.smem, pl.nunits),
                   STC_THREADS, pl.smem, st>>>(d, d.tc_synth, pl, d.legendre);
      const int eb = members_per_block(d.E, NP);
      k_synth_surf<<<dim3(NP, (d.E + eb - 1) / eb), 128, sm, st>>>(d, sp, eb);
      return;
    }
  }
  auto go = [&](auto kern) {
    if (attrs)
      allow_smem(kern);
    else
      kern<<<dim3(NP, (d.E + sp.eb - 1) / sp.eb, sp.nch + 1), sp.nt, sp.smem, st>>>(d, sp);
  };
  if constexpr (sizeof(R) == 4) {
    go(k_synth<R, 2, 2>);
  } else {
    if (sp.ntab == 3) go(k_synth<R, 2, 3>);
    else go(k_synth<R, 2, 2>);
  }
}
// Implicit update: 8- / 16-byte accesses where every complex array is so aligned.
template <typename R> void launch_implicit(const SD<R>& d, R dt, int set, int ra_mode,
                                           cudaStream_t st, bool attrs) {
  const ImplPlan pl = impl_plan(d.E, d.K, d.N);
  const int smem = (int)impl_smem<R>(d.K, pl.CC);
  const uintptr_t all = (uintptr_t)d.sa3 | (uintptr_t)d.sb3 | (uintptr_t)d.tend |
                        (uintptr_t)d.frc3;
  auto go = [&](auto kern) {
    if (attrs)
      allow_smem(kern);
    else
      kern<<<dim3((d.M + 1) / 2, d.E, pl.nch), pl.nt, smem, st>>>(d, dt, set, ra_mode, pl.CC);
  };
  if (all & (2 * sizeof(R) - 1)) go(k_implicit<R, false>);
  else go(k_implicit<R, true>);
}

// Grid of a persistent kernel: the CTAs that are resident at once on the
// current device (from the occupancy calculator, cached per kernel, block
// size, shared memory and device), at most `units`.
inline int persistent_grid(const void* fn, int nt, size_t smem, int units) {
  struct Entry { const void* fn; int nt, dev; size_t smem; int ctas; };
  static std::mutex mu;
  static Entry cache[32];
  static int ncache = 0;
  int dev = 0;
  cudaGetDevice(&dev);
  int ctas = 0;
  {
    std::lock_guard<std::mutex> lock(mu);
    for (int i = 0; i < ncache; ++i)
      if (cache[i].fn == fn && cache[i].nt == nt && cache[i].dev == dev && cache[i].smem == smem)
        ctas = cache[i].ctas;
    if (!ctas) {
      int sms = 0, per = 0;
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, nt, smem);
      ctas = (sms > 0 ? sms : 1) * (per > 0 ? per : 1);
      if (ncache < 32) cache[ncache++] = Entry{fn, nt, dev, smem, ctas};
    }
  }
  return ctas < units ? ctas : units;
}

template <int I> void launch_idft(const SD<float>& d, cudaStream_t st) {
  const size_t smem = idft_smem(I, d.M);
  const int nz = (idft_rows(d.K) + IDFT_RC - 1) / IDFT_RC;
  if (idft_chunks(d.E, d.J)) k_idft<I, true><<<dim3(d.J, d.E, nz), IDFT_NT, smem, st>>>(d, d.dft);
  else k_idft<I, false><<<dim3(d.J, d.E), IDFT_NT, smem, st>>>(d, d.dft);
}

template <typename R, int I, int BT, int MINB>
void launch_alg(const SD<R>& d, int ps_mode, cudaStream_t st, bool attrs) {
  const int LS = alg_seg<R>(d.E, d.J, I, d.K);
  if (!LS) {
    if (!attrs) k_alg<R, I, BT, MINB, false><<<dim3(d.J * (I / BT), d.E), BT, 0, st>>>(d, ps_mode, 0);
    return;
  }
  const int smem = 3 * 32 * (int)sizeof(R) * d.K;
  if (attrs)
    cudaFuncSetAttribute(k_alg<R, I, 32, 1, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         3 * 32 * (int)sizeof(R) * 64);
  else
    k_alg<R, I, 32, 1, true><<<dim3(d.J * (I / 32), d.E), 32 * ((d.K + LS - 1) / LS), smem, st>>>(
        d, ps_mode, LS);
}

template <typename R, int I> int launch_step(const SD<R>& d, const lbm_step_ctl& c,
                                             cudaStream_t st, int only = -1) {
  constexpr int KB = grid_kb<R, I>(), NT = grid_nt<R, I>();
  const int NP = (d.M + 1) / 2;
  const size_t gsm = GridSmem<R, I, KB, NT>::bytes(d.M);
  if constexpr (sizeof(R) == 4) {
    // grid-point part as three launches: longitude synthesis, column
    // algebra, longitude analysis (kernel ids 4, 5, 6; 0 = all three)
    if (only < 0 || only == 0 || only == 4)
      launch_idft<I>(d, st);
    if (only < 0 || only == 0 || only == 5)
      launch_alg<R, I, I, alg_minb<I>()>(d, c.ps_mode, st, false);
    if ((only < 0 || only == 0 || only == 6) && d.legendre && !(d.tc_off & 4) &&
        ftc_supported(I, d.K, d.N)) {
      const FtcPlan pl = ftc_plan(d.E, d.J, I, d.K, d.N);
      k_fdft_tc<<<persistent_grid((const void*)k_fdft_tc, FTC_THREADS, pl.smem, pl.nunits),
                  FTC_THREADS, pl.smem, st>>>(d, d.tc_dft, pl, d.legendre);
      // the surface rows on the FMA pipes; their FP32 cos table follows the
      // tensor-core image
      const float* cs = reinterpret_cast<const float*>(d.tc_dft + pl.tab_bytes);
      const int EB = fsurf_eb(d.E, d.J);
      const dim3 g(d.J, (d.E + EB - 1) / EB);
      if (EB == 2) k_fdft_surf<2><<<g, 128, fsurf_smem(I, 2), st>>>(d, cs);
      else k_fdft_surf<8><<<g, 128, fsurf_smem(I, 8), st>>>(d, cs);
    } else if (only < 0 || only == 0 || only == 6) {
      const FdftPlan pl = fdft_plan(I, d.M, d.K);
      const size_t smem = sizeof(float) * (size_t)pl.total;
      const int nunits = d.E * d.J * ((d.K + pl.lc - 1) / pl.lc);
      k_fdft<I><<<persistent_grid((const void*)k_fdft<I>, pl.nt, smem, nunits), pl.nt, smem,
                  st>>>(d, d.dft, pl);
    }
  } else if (only < 0 || only == 0) {
    if (d.grid6 && d.grid9) {
      // workspace for the grid rows: the grid part as three launches with
      // enough blocks for one member (1 member of T42L20 675 -> 145 us, 32
      // members 9.27 -> 2.95 ms)
      using G = GridFft<I>;
      k_ifft<R, I><<<dim3(d.J, 1 + (d.K + G::LI - 1) / G::LI, d.E), G::NTI,
                     G::template ifft_smem<R>(d.M), st>>>(d);
      launch_alg<R, I, 32, 1>(d, c.ps_mode, st, false);
      k_ffft<R, I><<<dim3(d.J, 1 + (d.K + G::LF - 1) / G::LF, d.E), G::NTF,
                     G::template ffft_smem<R>(d.M), st>>>(d);
    } else {
      k_grid<R, I, KB, NT><<<dim3(d.J, d.E), NT, gsm, st>>>(d, c.ps_mode);
    }
  }
  if (only < 0 || only == 1) {
    if constexpr (sizeof(R) == 4) {
      if (d.legendre && !(d.tc_off & 1)) {
        const AtcPlan pl = atc_plan(d.E, d.J, d.K, d.N, d.tc_g);
        k_anal_tc<<<persistent_grid((const void*)k_anal_tc, ATC_THREADS, pl.smem, pl.nunits),
                    ATC_THREADS, pl.smem, st>>>(d, d.tc_anal, pl, d.legendre);
      }
    }
    bool level = true;
    if constexpr (sizeof(R) == 4) {
      if (d.legendre && !(d.tc_off & 1)) {
        const int eb = members_per_block(d.E, NP);
        k_anal_surf<<<dim3(NP, (d.E + eb - 1) / eb), 128, anal_surf_smem(d.J, d.N), st>>>(d, eb);
        level = false;
      }
    }
    if (level) launch_anal<R>(d, st, false);
  }
  if (only < 0 || only == 2)
    launch_implicit<R>(d, R(c.dt), c.set, c.ra_mode, st, false);
  if (only < 0 || only == 3) launch_synth<R>(d, st, false);
  LBM_LAUNCH_CHECK();
  return LBM_OK;
}

template <typename R, int I> void set_attrs(const SD<R>& d) {
  constexpr int KB = grid_kb<R, I>(), NT = grid_nt<R, I>();
  launch_alg<R, I, sizeof(R) == 4 ? I : 32, sizeof(R) == 4 ? alg_minb<I>() : 1>(d, 0, 0, true);
  if constexpr (sizeof(R) == 4) {
    allow_smem(k_idft<I, false>);
    allow_smem(k_idft<I, true>);
    const FdftPlan pl = fdft_plan(I, d.M, d.K);
    const size_t smem = sizeof(float) * (size_t)pl.total;
    if (smem <= 227 * 1024) {
      allow_smem(k_fdft<I>);
      persistent_grid((const void*)k_fdft<I>, pl.nt, smem, 1);
    }
    if (d.legendre && ftc_supported(I, d.K, d.N)) {
      const FtcPlan fp = ftc_plan(d.E, d.J, I, d.K, d.N);
      allow_smem(k_fdft_tc);
      persistent_grid((const void*)k_fdft_tc, FTC_THREADS, fp.smem, 1);
    }
  } else {
    allow_smem(k_grid<R, I, KB, NT>);
    allow_smem(k_ifft<R, I>);
    allow_smem(k_ffft<R, I>);
  }
  launch_anal<R>(d, nullptr, true);
  launch_synth<R>(d, nullptr, true);
  if constexpr (sizeof(R) == 4) {
    if (d.legendre) {
      const AtcPlan pl = atc_plan(d.E, d.J, d.K, d.N, d.tc_g);
      allow_smem(k_anal_tc);
      allow_smem(k_anal_surf);
      persistent_grid((const void*)k_anal_tc, ATC_THREADS, pl.smem, 1);
    }
  }
  launch_implicit<R>(d, R(0), 0, 0, nullptr, true);
  if constexpr (sizeof(R) == 4) {
    if (d.legendre) {
      const StcPlan pl = stc_plan(d.E, d.J, d.K, d.N, d.tc_g);
      allow_smem(k_synth_tc);
      persistent_grid((const void*)k_synth_tc, STC_THREADS, pl.smem, 1);
    }
  }
}

template <typename R> int validate(const SD<R>& d) {
  if (d.E < 1 || d.K < 1 || d.K > 64 || d.N < 1 || (d.J & 1) || 2 * d.M > d.I) return LBM_ERR_ARG;
  if (d.I != 64 && d.I != 128 && d.I != 256) return LBM_ERR_ARG;
  if (IM_THREADS / d.K < 1) return LBM_ERR_ARG;
  if (!d.symp || !d.symh || !d.tw || !d.jfac || !d.vert || !d.b3 || !d.bsd || !d.b2 ||
      !d.lap || !d.invlap || !d.nn1a || !d.kv || !d.kd || !d.ktt || !d.kq ||
      !d.minv || !d.sa3 || !d.sas || !d.sb3 || !d.psa || !d.psb || !d.sf ||
      !d.sfs || !d.af || !d.afs || !d.tend || !d.tends || !d.err)
    return LBM_ERR_ARG;
  for (int f = 0; f < 4; ++f)
    if (d.vd_on[f] && !d.vdiff) return LBM_ERR_ARG;
  if (sizeof(R) == 4 && (!d.dft || !d.grid6 || !d.grid9)) return LBM_ERR_ARG;
  // 16-byte copies and bulk prefetches read sf, af and grid9, the tensor-core
  // synthesis sa3; FP32 pairs in one access: sfs, dft and (k_fdft) afs
  auto off = [](const void* p, int n) { return ((uintptr_t)p & (n - 1)) != 0; };
  if (off(d.sf, 16) || off(d.af, 16) || (sizeof(R) == 4 && off(d.grid9, 16))) return LBM_ERR_ARG;
  if (sizeof(R) == 4) {
    const bool tc_dft = d.legendre && !(d.tc_off & 4) && ftc_supported(d.I, d.K, d.N);
    if (off(d.sfs, 8) || off(d.dft, 8) || (!tc_dft && off(d.afs, 8)) ||
        (d.legendre && !(d.tc_off & 2) && off(d.sa3, 16)))
      return LBM_ERR_ARG;
  }
  if (d.legendre) {
    // tensor-core analysis: FP32 state, 16-latitude steps, 16-byte af rows,
    // at most 256 table rows, the plan within shared memory
    if (sizeof(R) != 4 || (d.legendre != 3 && d.legendre != 6) || !d.tc_anal ||
        !d.tc_synth || (d.J % 16) || (d.K & 1) || d.M > 256 ||
        atc_plan(d.E, d.J, d.K, d.N, d.tc_g).smem > 227 * 1024 ||
        stc_plan(d.E, d.J, d.K, d.N, d.tc_g).smem > 227 * 1024 ||
        (stc_plan(d.E, d.J, d.K, d.N).JT % 16) || d.tc_off < 0 || d.tc_off > 7 ||
        d.tc_g < 0 ||
        (ftc_supported(d.I, d.K, d.N) &&
         (!d.tc_dft || ((uintptr_t)d.tc_dft & 15) ||
          ftc_plan(d.E, d.J, d.I, d.K, d.N).smem > 227 * 1024)) ||
        ((uintptr_t)d.tc_anal & 15) || ((uintptr_t)d.tc_synth & 15))
      return LBM_ERR_ARG;
  }
  if (sizeof(R) == 4 &&
      (idft_smem(d.I, d.M) > 227 * 1024 ||
       sizeof(float) * (size_t)fdft_plan(d.I, d.M, d.K).total > 227 * 1024))
    return LBM_ERR_ARG;
  return LBM_OK;
}

template <typename R> int run_steps(const lbm_stepper_desc* desc, const lbm_step_ctl* ctl,
                                    int nsteps, cudaStream_t st) {
  const SD<R> d = make_sd<R>(*desc);
  int rc = validate(d);
  if (rc) return rc;
  for (int s = 0; s < nsteps; ++s) {
    if (ctl[s].set < 0 || ctl[s].set >= d.nsets) return LBM_ERR_ARG;
    switch (d.I) {
      case 64: rc = launch_step<R, 64>(d, ctl[s], st); break;
      case 128: rc = launch_step<R, 128>(d, ctl[s], st); break;
      default: rc = launch_step<R, 256>(d, ctl[s], st); break;
    }
    if (rc) return rc;
  }
  return LBM_OK;
}

template <typename R> int launch_one(const lbm_stepper_desc* desc, const lbm_step_ctl& c,
                                     int kernel, cudaStream_t st) {
  const SD<R> d = make_sd<R>(*desc);
  int rc = validate(d);
  if (rc) return rc;
  if (c.set < 0 || c.set >= d.nsets) return LBM_ERR_ARG;
  switch (d.I) {
    case 64: return launch_step<R, 64>(d, c, st, kernel);
    case 128: return launch_step<R, 128>(d, c, st, kernel);
    default: return launch_step<R, 256>(d, c, st, kernel);
  }
}

// Whether the plans of the Legendre kernels in use and of the implicit update fit a
// block's shared memory (those of the other kernels: validate).
template <typename R> bool plans_fit(const SD<R>& d) {
  const size_t most = 227 * 1024;
  const bool tc_anal = d.legendre && !(d.tc_off & 1), tc_synth = d.legendre && !(d.tc_off & 2);
  const SynthPlan sp = synth_plan<R>(d.E, d.J, d.K, d.N);
  const size_t anal = tc_anal ? anal_surf_smem(d.J, d.N)
                              : anal_plan<R>(d.E, d.J, d.K, d.N).smem;
  const size_t synth = tc_synth ? sp.ox + sizeof(C2<R>) * 4 * (d.N + 2) : sp.smem;
  return anal <= most && synth <= most &&
         impl_smem<R>(d.K, impl_plan(d.E, d.K, d.N).CC) <= most;
}

template <typename R> int prepare_attrs(const lbm_stepper_desc* desc) {
  const SD<R> d = make_sd<R>(*desc);
  int rc = validate(d);
  if (rc) return rc;
  if (!plans_fit(d)) return LBM_ERR_ARG;
  switch (d.I) {
    case 64: set_attrs<R, 64>(d); break;
    case 128: set_attrs<R, 128>(d); break;
    default: set_attrs<R, 256>(d); break;
  }
  return cudaGetLastError() == cudaSuccess ? LBM_OK : LBM_ERR_LAUNCH;
}

template <typename R> int prime(const lbm_stepper_desc* desc, cudaStream_t st) {
  const SD<R> d = make_sd<R>(*desc);
  int rc = validate(d);
  if (rc) return rc;
  launch_synth<R>(d, st, false);
  LBM_LAUNCH_CHECK();
  return LBM_OK;
}

template <typename R> int colsum(const lbm_stepper_desc* desc, cudaStream_t st) {
  const SD<R> d = make_sd<R>(*desc);
  int rc = validate(d);
  if (rc) return rc;
  k_colsum<R><<<dim3((d.NS + 127) / 128, d.E), 128, 0, st>>>(d);
  LBM_LAUNCH_CHECK();
  return LBM_OK;
}

template <typename R> int flush(const lbm_stepper_desc* desc, int ps_mode, cudaStream_t st) {
  const SD<R> d = make_sd<R>(*desc);
  int rc = validate(d);
  if (rc) return rc;
  switch (d.I) {
    case 64: k_ps_flush<R, 64><<<dim3(d.J, d.E), FftShape<64>::R1, 0, st>>>(d, ps_mode); break;
    case 128: k_ps_flush<R, 128><<<dim3(d.J, d.E), FftShape<128>::R1, 0, st>>>(d, ps_mode); break;
    default: k_ps_flush<R, 256><<<dim3(d.J, d.E), FftShape<256>::R1, 0, st>>>(d, ps_mode); break;
  }
  LBM_LAUNCH_CHECK();
  return LBM_OK;
}

// ---- stepping from a static scratch area ------------------------------------
// lbm_stepper_run_noalloc takes the intermediate buffers of a step (sf, sfs,
// af, afs, tend, tends and in FP32 mode grid6, grid9) from this file-scope
// array instead of caller memory.  It is sized once, at LBM_NOALLOC_SCRATCH_BYTES, and every GPU that
// loads the library holds it until the process exits.
static __device__ __align__(256) unsigned char g_noalloc_scratch[LBM_NOALLOC_SCRATCH_BYTES];

constexpr int NOALLOC_MAX_DEVICES = 64;
static std::mutex g_noalloc_mu;
static void* g_noalloc_base[NOALLOC_MAX_DEVICES];

// Byte offsets of sf, sfs, af, afs, tend, tends (and with `rows` grid6, grid9)
// in the scratch area, each rounded up to 256 bytes.  `need` is the total,
// computed in double so that an absurd size cannot wrap around before it is
// compared with the maximum.
static void noalloc_layout(const lbm_stepper_desc& d, bool rows, size_t off[8], double* need) {
  const double c = 2.0 * (d.prec == LBM_F64 ? sizeof(double) : sizeof(float));
  const double E = d.nmem, M = d.nmax + 1.0, J = d.nlat, K = d.kmax, I = d.nlon;
  const double NS = M * (M + 1.0) / 2.0;
  const double r = rows ? 0.5 * c : 0.0;
  const double bytes[8] = {c * E * M * J * K * 6, c * E * M * J * 5, c * E * M * J * K * 7,
                           c * E * M * J * 2,     c * E * 4 * NS * K, c * E * 2 * NS,
                           r * E * J * (6 + 6 * K) * I, r * E * J * (2 + 9 * K) * I};
  double t = 0.0;
  for (int i = 0; i < 8; ++i) {
    off[i] = (size_t)t;
    t += 256.0 * std::ceil(bytes[i] / 256.0);
  }
  *need = t;
}

// Device address of the scratch area on the current device.  The first call
// on a device looks it up with cudaGetSymbolAddress (with that device
// current) and keeps it; later calls reuse it.  The address belongs to the
// device's primary context (the one the CUDA runtime uses): a caller running
// under another context of its own, or one that resets the device after the
// first call, would be handed an address that is no longer valid there.
static int noalloc_base(void** out) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NOALLOC_MAX_DEVICES)
    return LBM_ERR_LAUNCH;
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (!g_noalloc_base[dev]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) return LBM_ERR_LAUNCH;
    g_noalloc_base[dev] = p;
  }
  *out = g_noalloc_base[dev];
  return LBM_OK;
}

template <typename R> int run_noalloc(const lbm_stepper_desc& w, const lbm_step_ctl* ctl,
                                      int nsteps, size_t clear, cudaStream_t st) {
  // the full argument check runs before the clear, capturing or not
  const int vrc = validate(make_sd<R>(w));
  if (vrc) return vrc;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  cudaStreamIsCapturing(st, &cs);
  if (cs == cudaStreamCaptureStatusNone) {
    const int rc = prepare_attrs<R>(&w);
    if (rc) return rc;
  }
  if (cudaMemsetAsync(w.sf, 0, clear, st) != cudaSuccess) return LBM_ERR_LAUNCH;
  const int rc = prime<R>(&w, st);
  if (rc) return rc;
  return run_steps<R>(&w, ctl, nsteps, st);
}

}  // namespace lbm

using namespace lbm;

struct lbm_graph {
  cudaGraph_t graph;
  cudaGraphExec_t exec;
};

extern "C" {

int lbm_stepper_prime(const lbm_stepper_desc* d, void* stream) {
  if (!d) return LBM_ERR_ARG;
  int rc = d->prec == LBM_F64 ? prepare_attrs<double>(d) : prepare_attrs<float>(d);
  if (rc) return rc;
  return d->prec == LBM_F64 ? prime<double>(d, (cudaStream_t)stream)
                            : prime<float>(d, (cudaStream_t)stream);
}

int lbm_stepper_run(const lbm_stepper_desc* d, const lbm_step_ctl* ctl, int nsteps,
                    void* stream) {
  if (!d || !ctl || nsteps < 0 || (d->prec != LBM_F64 && d->prec != LBM_F32)) return LBM_ERR_ARG;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  cudaStreamIsCapturing((cudaStream_t)stream, &cs);
  if (cs == cudaStreamCaptureStatusNone) {
    int rc = d->prec == LBM_F64 ? prepare_attrs<double>(d) : prepare_attrs<float>(d);
    if (rc) return rc;
  }
  return d->prec == LBM_F64 ? run_steps<double>(d, ctl, nsteps, (cudaStream_t)stream)
                            : run_steps<float>(d, ctl, nsteps, (cudaStream_t)stream);
}

int lbm_stepper_launch(const lbm_stepper_desc* d, const lbm_step_ctl* ctl, int kernel,
                       void* stream) {
  if (!d || !ctl || kernel < 0 || kernel > 6 || (d->prec != LBM_F64 && d->prec != LBM_F32) ||
      (kernel > 3 && d->prec != LBM_F32))
    return LBM_ERR_ARG;
  int rc = d->prec == LBM_F64 ? prepare_attrs<double>(d) : prepare_attrs<float>(d);
  if (rc) return rc;
  return d->prec == LBM_F64 ? launch_one<double>(d, *ctl, kernel, (cudaStream_t)stream)
                            : launch_one<float>(d, *ctl, kernel, (cudaStream_t)stream);
}

int lbm_stepper_flush(const lbm_stepper_desc* d, int ps_mode, void* stream) {
  if (!d || ps_mode < 0 || ps_mode > 2) return LBM_ERR_ARG;
  return d->prec == LBM_F64 ? flush<double>(d, ps_mode, (cudaStream_t)stream)
                            : flush<float>(d, ps_mode, (cudaStream_t)stream);
}

int lbm_stepper_colsum(const lbm_stepper_desc* d, void* stream) {
  if (!d) return LBM_ERR_ARG;
  return d->prec == LBM_F64 ? colsum<double>(d, (cudaStream_t)stream)
                            : colsum<float>(d, (cudaStream_t)stream);
}

int lbm_graph_capture(const lbm_stepper_desc* d, const lbm_step_ctl* ctl, int nsteps,
                      void* stream, lbm_graph** out) {
  if (!d || !ctl || !out || nsteps < 1) return LBM_ERR_ARG;
  int rc = d->prec == LBM_F64 ? prepare_attrs<double>(d) : prepare_attrs<float>(d);
  if (rc) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  if (cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) != cudaSuccess)
    return LBM_ERR_LAUNCH;
  rc = d->prec == LBM_F64 ? run_steps<double>(d, ctl, nsteps, st)
                          : run_steps<float>(d, ctl, nsteps, st);
  cudaGraph_t g = nullptr;
  const cudaError_t ec = cudaStreamEndCapture(st, &g);
  if (rc || ec != cudaSuccess || !g) {
    if (g) cudaGraphDestroy(g);
    return rc ? rc : LBM_ERR_LAUNCH;
  }
  cudaGraphExec_t ex = nullptr;
  if (cudaGraphInstantiate(&ex, g, 0) != cudaSuccess) {
    cudaGraphDestroy(g);
    return LBM_ERR_LAUNCH;
  }
  lbm_graph* h = new (std::nothrow) lbm_graph;
  if (!h) {
    cudaGraphExecDestroy(ex);
    cudaGraphDestroy(g);
    return LBM_ERR_LAUNCH;
  }
  h->graph = g;
  h->exec = ex;
  *out = h;
  return LBM_OK;
}

int lbm_graph_launch(lbm_graph* g, void* stream) {
  if (!g) return LBM_ERR_ARG;
  return cudaGraphLaunch(g->exec, (cudaStream_t)stream) == cudaSuccess ? LBM_OK
                                                                       : LBM_ERR_LAUNCH;
}

int lbm_graph_destroy(lbm_graph* g) {
  if (!g) return LBM_ERR_ARG;
  cudaGraphExecDestroy(g->exec);
  cudaGraphDestroy(g->graph);
  delete g;
  return LBM_OK;
}

int lbm_stepper_run_noalloc(const lbm_stepper_desc* d, const lbm_step_ctl* ctl, int nsteps,
                            void* stream) {
  if (!d || !ctl || nsteps < 0 || (d->prec != LBM_F64 && d->prec != LBM_F32)) return LBM_ERR_ARG;
  if (d->nmem < 1 || d->nlat < 2 || d->nmax < 1 || d->kmax < 1) return LBM_ERR_ARG;
  if (d->nlon != 64 && d->nlon != 128 && d->nlon != 256) return LBM_ERR_ARG;
  size_t off[8];
  double need = 0.0;
  // FP32 needs the grid rows; FP64 takes them (the split grid part) where the
  // scratch area has room, and runs k_grid otherwise
  bool rows = true;
  noalloc_layout(*d, rows, off, &need);
  if (d->prec == LBM_F64 && need > (double)LBM_NOALLOC_SCRATCH_BYTES) {
    rows = false;
    noalloc_layout(*d, rows, off, &need);
  }
  if (!(need > 0.0)) return LBM_ERR_ARG;
  if (need > (double)LBM_NOALLOC_SCRATCH_BYTES) return LBM_ERR_SCRATCH;
  for (int s = 0; s < nsteps; ++s)
    if (ctl[s].set < 0 || ctl[s].set >= d->nsets || ctl[s].ps_mode < 0 || ctl[s].ps_mode > 2 ||
        ctl[s].ra_mode < 0 || ctl[s].ra_mode > 1)
      return LBM_ERR_ARG;
  void* base = nullptr;
  const int rc = noalloc_base(&base);
  if (rc) return rc;
  unsigned char* b = static_cast<unsigned char*>(base);
  lbm_stepper_desc w = *d;
  w.sf = b + off[0];
  w.sfs = b + off[1];
  w.af = b + off[2];
  w.afs = b + off[3];
  w.tend = b + off[4];
  w.tends = b + off[5];
  w.grid6 = rows ? b + off[6] : nullptr;
  w.grid9 = rows ? b + off[7] : nullptr;
  const size_t clear = (size_t)need;
  cudaStream_t st = (cudaStream_t)stream;
  return d->prec == LBM_F64 ? run_noalloc<double>(w, ctl, nsteps, clear, st)
                            : run_noalloc<float>(w, ctl, nsteps, clear, st);
}

}  // extern "C"
