// Implicit spectral update of the step (included by stepper.cu after
// legendre_fma.cuh).
#pragma once

namespace lbm {

constexpr int IM_THREADS = 256;

// Coefficients per block and blocks per n-pair: an even share of the N + 2
// coefficients of a pair, at most IM_THREADS / K of them; small ensembles take
// smaller shares (down to four) until there are two blocks per SM.
struct ImplPlan { int CC, nch, nt; };
inline ImplPlan impl_plan(int E, int K, int N) {
  const int NP = (N + 2) / 2, most = IM_THREADS / K, nco = N + 2;
  int nch = (nco + most - 1) / most;
  while (NP * E * nch < 2 * FILL_SMS && (nco + nch) / (nch + 1) >= 4) ++nch;
  ImplPlan p;
  p.CC = (nco + nch - 1) / nch;
  p.nch = (nco + p.CC - 1) / p.CC;
  p.nt = (p.CC * K + 31) / 32 * 32;
  return p;
}
// Operators (minv of two n, vertical diffusion, level factors) and seven exchanges.
template <typename R> size_t impl_smem(int K, int CC) {
  return sizeof(R) * ((size_t)(2 + 4) * K * K + 7 * (size_t)K + (K & 1)) +
         sizeof(C2<R>) * 7 * (size_t)CC * K;
}

// The semi-implicit update in the order of integrator.py:264-315.  Three
// places subtract nearly equal quantities, and the FP32 mode carries them in
// float-float (XF) so that the difference keeps FP32 relative precision:
// the divergence right-hand side (explicit tendency against the Laplacian of
// the geopotential), the temperature update (heating against the
// reference-temperature matrix on the mean divergence) and the pi update
// (against the column-integrated divergence).  WW and tmtx enter through
// their level-scan forms
//   (WW x)_k   = R alpha_k x_k + sum_{l<k} R dlog3_l x_l,
//   (tmtx D)_k = kappa Tref_k (alpha_k D_k + w3_k sum_{l>k} dsig_l D_l),
// each level summing its own prefix / suffix.  Damping factors 1 / (1 + c)
// are applied as x - x c / (1 + c) so that a small c keeps its precision.
//
// Block (n-pair, member, share of the pair's coefficients), one thread per
// (coefficient, level), one buffer per exchange: four barriers (five with
// vertical diffusion) in all.  The time goes into the compensated sum of M(n)^-1
// rhs (26 FP32 operations per term) and into the latency of the loads, so the
// blocks are short and many: a block that walked all coefficients of a pair, with
// twelve barriers each time, left one member of T42L20 on 22 SMs.  NAT: the
// complex arrays are aligned to their element size (8- / 16-byte accesses).
// us at T42L20 before -> after: FP32 1 member 29 -> 11, 128 members 213 -> 177, 512
// members 801 -> 686; FP64 1 member 135 -> 30, 32 members 519 -> 317.  (Packed pairs
// for the sums save issue slots but spill at 80 registers: 207 at 128 members.)
template <typename R, bool NAT> LBM_D C2<R> ldn(const C2<R>* p) {
  if constexpr (NAT) return ldc(p);
  else return *p;
}
template <typename R, bool NAT> LBM_D void stn(C2<R>* p, C2<R> a) {
  if constexpr (NAT) stc(p, a);
  else *p = a;
}
template <typename R, bool NAT>
__global__ void __launch_bounds__(IM_THREADS, sizeof(R) == 4 ? 3 : 2)
    k_implicit(SD<R> d, R dt, int set, int ra_mode, int CC) {
  const int p = blockIdx.x, e = blockIdx.y, c0 = blockIdx.z * CC;
  const int K = d.K, N = d.N, NS = d.NS;
  const int n1 = p, n2 = N - p;
  const int C1 = n1 + 1, C2n = (n2 != n1) ? n2 + 1 : 0;
  const int ncoef = C1 + C2n;
  if (c0 >= ncoef) return;                      // the middle pair of an even N is one n
  extern __shared__ __align__(16) unsigned char smraw[];
  R* mi = reinterpret_cast<R*>(smraw);          // [2][K][K] minv^T (l, k)
  R* vdT = mi + 2 * K * K;                      // [4][K][K] (vdiff - I)^T (l, k)
  R* vs = vdT + 4 * K * K;                      // [6][K] RALPHA RDLOG3 GG DSIG ALPHA W3
  R* ktr = vs + 6 * K;                          // [K] KTREF
  C2<R>* bA = reinterpret_cast<C2<R>*>(ktr + K + (K & 1));  // [7][CC][K]
  const int tid = threadIdx.x, nt = blockDim.x, CK = CC * K;
  const R dt2 = R(2) * dt, gam = d.robert;
  const C2<R> z = cmk<R>(0, 0);
  const size_t e3 = (size_t)e * 4 * NS * K, F = (size_t)NS * K;
  const size_t efrc3 = d.frc_shared ? 0 : e3;
  const size_t efrcs = d.frc_shared ? 0 : (size_t)e * NS;
  // ---- this thread's coefficient and level, and its values (loads first)
  const FastDiv fK(K);
  const int c = fK.div(tid), k = tid - c * K;
  const int coef = c0 + c;
  const bool act = (c < CC) && (coef < ncoef);
  int n = 0, m = 0, sel = 0;
  if (act) {
    if (coef < C1) { n = n1; m = coef; sel = 0; }
    else { n = n2; m = coef - C1; sel = 1; }
  }
  const size_t idx = (size_t)spec_index(m, n, N);
  const size_t o = idx * K + k;
  C2<R> aV = z, aD = z, aT = z, aQ = z, bV = z, bD = z, bT = z, bQ = z;
  C2<R> wV = z, wD = z, wT = z, wQ = z, wpi = z, pp = z;
  R ktt = 0, kd = 0, kv = 0, kq = 0, lap = 0;
  if (act) {
    auto L = [](const C2<R>* q) { return ldn<R, NAT>(q); };
    bT = L(d.sb3 + e3 + 2 * F + o); wT = L(d.tend + e3 + 2 * F + o);
    bD = L(d.sb3 + e3 + 1 * F + o); wD = L(d.tend + e3 + 1 * F + o);
    wpi = d.tends[((size_t)e * 2 + 0) * NS + idx];
    pp = d.tends[((size_t)e * 2 + 1) * NS + idx];
    bV = L(d.sb3 + e3 + 0 * F + o); wV = L(d.tend + e3 + 0 * F + o);
    bQ = L(d.sb3 + e3 + 3 * F + o); wQ = L(d.tend + e3 + 3 * F + o);
    aV = L(d.sa3 + e3 + 0 * F + o); aD = L(d.sa3 + e3 + 1 * F + o);
    aT = L(d.sa3 + e3 + 2 * F + o); aQ = L(d.sa3 + e3 + 3 * F + o);
    if (d.frc3) {
      wV = wV + L(d.frc3 + efrc3 + 0 * F + o); wD = wD + L(d.frc3 + efrc3 + 1 * F + o);
      wT = wT + L(d.frc3 + efrc3 + 2 * F + o); wQ = wQ + L(d.frc3 + efrc3 + 3 * F + o);
    }
    if (d.frcs) wpi = wpi + d.frcs[efrcs + idx];
    ktt = d.ktt[n * K + k]; kd = d.kd[n * K + k]; kv = d.kv[n * K + k]; kq = d.kq[n * K + k];
    lap = d.lap[n];
  }
  // ---- operators of the n's of this share
  const R* mset = d.minv + (size_t)set * d.M * K * K;
  for (int x = tid; x < K * K; x += nt) {
    if (c0 < C1) mi[x] = mset[(size_t)n1 * K * K + x];
    if (c0 + CC > C1) mi[K * K + x] = mset[(size_t)n2 * K * K + x];
  }
  for (int f = 0; f < 4; ++f)
    if (d.vd_on[f])
      for (int x = tid; x < K * K; x += nt)
        vdT[f * K * K + x] = d.vdiff[((size_t)set * 4 + f) * K * K + x];
  for (int x = tid; x < K; x += nt) {
    vs[0 * K + x] = vrow(d, LBM_VERT_RALPHA, x);
    vs[1 * K + x] = vrow(d, LBM_VERT_RDLOG3, x);
    vs[2 * K + x] = vrow(d, LBM_VERT_GG, x);
    vs[3 * K + x] = vrow(d, LBM_VERT_DSIG, x);
    vs[4 * K + x] = vrow(d, LBM_VERT_ALPHA, x);
    vs[5 * K + x] = vrow(d, LBM_VERT_W3, x);
    ktr[x] = vrow(d, LBM_VERT_KTREF, x);
  }
  C2<R>* A = bA + c * K;                        // exchange q of this coefficient: A + q CK
  const R bt = dt2 * ktt;                       // 2 dt ktt; ft = 1 + bt
  // wdx = T(t-dt) (1 + dt ktt) + dt wT  (integrator.py:287)
  if (act) stc(A + k, bT + (bT * ktt + wT) * dt);
  __syncthreads();
  if (act) {
    C2<R> pre = z;                                       // sum_{l<k} R dlog3_l wdx_l
#pragma unroll 4
    for (int l = 0; l < k; ++l) cfma(pre, vs[1 * K + l], ldc(A + l));
    CX<R> phi = cx_add(cx_prod(vs[0 * K + k], ldc(A + k)), cx(pre));   // WW wdx
    const C2<R> wdpix = pp + wpi * dt;
    const R gk = vs[2 * K + k];
    // wdphiy = WW wdx + ft gg wdpix, ft gg taken as gg + bt gg
    phi = cx_add(phi, cx_add(cx_prod(gk, wdpix), cx_mul(cx_prod(bt, wdpix), gk)));
    // dt (wD ft - lap wdphiy), the two terms nearly balancing
    const CX<R> zz = cx_add(cx_add(cx(wD), cx_prod(bt, wD)), cx_mul(phi, -lap));
    const R ad = dt * kd;
    stc(A + CK + k, bD + (bD * (ad + bt + ad * bt) + cx_val(zz) * dt));
  }
  __syncthreads();
  C2<R> dbar = z;
  if (act) {
    const R* mm_ = mi + sel * K * K + k;
    const C2<R>* B = A + CK;
    // M(n)^-1 rhs with exact products and compensated sums (the divergence
    // of a balanced flow is small against the terms of this sum)
    CX<R> acc = cx<R>(z);
#pragma unroll 4
    for (int l = 0; l < K; ++l) acc = cx_add(acc, cx_prod(mm_[l * K], ldc(B + l)));   // minv (l, k)
    dbar = cx_val(acc);
    stc(A + 2 * CK + k, dbar);
  }
  __syncthreads();
  C2<R> nV = z, nD = z, nT = z, nQ = z, npi = z;
  if (act) {
    const C2<R>* D = A + 2 * CK;
    C2<R> suf = z;                                        // sum_{l>k} dsig_l dbar_l
#pragma unroll 4
    for (int l = K - 1; l > k; --l) cfma(suf, vs[3 * K + l], ldc(D + l));
    const CX<R> sfx = cx(suf);
    const CX<R> corr = cx_mul(cx_add(cx_prod(vs[4 * K + k], dbar), cx_mul(sfx, vs[5 * K + k])),
                              ktr[k]);
    const C2<R> yT = bT + cx_val(cx_add(cx(wT), cx_neg(corr))) * dt2;
    nT = yT - yT * (bt / (R(1) + bt));
    if (k == 0) {
      const CX<R> dsum = cx_add(sfx, cx_prod(vs[3 * K], dbar));
      npi = pp + cx_val(cx_add(cx(wpi), cx_neg(dsum))) * dt2;
    }
    nD = dbar * R(2) - bD;
    const R av = dt2 * kv, aq = dt2 * kq;
    const C2<R> xV = bV + wV * dt2, xQ = bQ + wQ * dt2;
    nV = xV - xV * (av / (R(1) + av));
    nQ = xQ - xQ * (aq / (R(1) + aq));
  }
  // implicit vertical diffusion (integrator.py:311-314); vdT holds the
  // operator minus the identity
  if (d.vd_on[0] || d.vd_on[1] || d.vd_on[2] || d.vd_on[3]) {
    C2<R>* vals[4] = {&nV, &nD, &nT, &nQ};
#pragma unroll
    for (int f = 0; f < 4; ++f)
      if (act && d.vd_on[f]) stc(A + (3 + f) * CK + k, *vals[f]);
    __syncthreads();
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      if (act && d.vd_on[f] && !(f < 2 && n < 2)) {
        C2<R> o2 = *vals[f];
        const R* vm = vdT + f * K * K + k;
        const C2<R>* X = A + (3 + f) * CK;
#pragma unroll 4
        for (int l = 0; l < K; ++l) cfma(o2, vm[l * K], ldc(X + l));
        *vals[f] = o2;
      }
    }
  }
  // column sums for sigma-dot of the next step (the first two exchanges are free)
  if (act) {
    stc(A + k, nV);
    stc(A + CK + k, nD);
  }
  // Robert-Asselin filter of the previous level (spectral part) and update
  if (act) {
    C2<R> fV, fD, fT, fQ;
    if (ra_mode) {
      fV = aV + (bV - aV * R(2) + nV) * gam;
      fD = aD + (bD - aD * R(2) + nD) * gam;
      fT = aT + (bT - aT * R(2) + nT) * gam;
      fQ = aQ + (bQ - aQ * R(2) + nQ) * gam;
    } else {
      fV = aV; fD = aD; fT = aT; fQ = aQ;
    }
    stn<R, NAT>(d.sb3 + e3 + 0 * F + o, fV); stn<R, NAT>(d.sb3 + e3 + 1 * F + o, fD);
    stn<R, NAT>(d.sb3 + e3 + 2 * F + o, fT); stn<R, NAT>(d.sb3 + e3 + 3 * F + o, fQ);
    stn<R, NAT>(d.sa3 + e3 + 0 * F + o, nV); stn<R, NAT>(d.sa3 + e3 + 1 * F + o, nD);
    stn<R, NAT>(d.sa3 + e3 + 2 * F + o, nT); stn<R, NAT>(d.sa3 + e3 + 3 * F + o, nQ);
    const bool fin = isfinite(nV.x) && isfinite(nV.y) && isfinite(nD.x) && isfinite(nD.y) &&
                     isfinite(nT.x) && isfinite(nT.y) && isfinite(nQ.x) && isfinite(nQ.y) &&
                     isfinite(npi.x) && isfinite(npi.y);
    if (!fin) {
      atomicOr(d.err, 1);
      if (d.err_member) atomicOr(d.err_member + e, 1);
    }
  }
  __syncthreads();
  // two threads per coefficient, all in the first warps: vorticity, divergence
  if (k == 0 && act) d.sas[(size_t)e * 4 * NS + idx] = npi;
  for (int x = tid; x < 2 * CC; x += nt) {
    const int cc = x >> 1, co = c0 + cc, w = x & 1;
    if (co >= ncoef) break;
    const int nn = co < C1 ? n1 : n2, mm = co < C1 ? co : co - C1;
    const C2<R>* X = bA + w * CK + cc * K;
    C2<R> v = z;
#pragma unroll 4
    for (int l = 0; l < K; ++l) cfma(v, vs[3 * K + l], ldc(X + l));
    const R il = d.invlap[nn];
    C2<R>* o2 = d.sas + (size_t)e * 4 * NS + spec_index(mm, nn, N);
    if (w == 0) {
      o2[NS] = v * il;                        // sum dsig psi
    } else {
      o2[2 * (size_t)NS] = v * il;            // sum dsig chi
      o2[3 * (size_t)NS] = v;                 // sum dsig div
    }
  }
}

}  // namespace lbm
