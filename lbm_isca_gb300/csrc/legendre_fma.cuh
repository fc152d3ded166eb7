// Legendre contractions of the step on the FMA pipes (included by stepper.cu):
// k_anal (af, afs -> tend, tends) and k_synth (state -> sf, sfs), FP32 and
// FP64, and their surface-only forms for the tensor-core placements.
//
// Both are small matrix products per pair of wavenumbers (m, N - m), whose
// N + 2 rows balance the triangle.  A row's parity (n - m even or odd) decides
// which equatorially symmetric or antisymmetric part it meets, so threads own
// rows of ONE parity: k_anal a tile of RT such rows at one level, k_synth JG
// latitudes at one level for the even or the odd rows (the two lanes of a
// latitude exchange their sums at the end, one writes the north, the other the
// south).  Each value read from shared memory then feeds twice the products of
// a thread that walks both parities, and the north +- south sums are formed
// once, when k_anal stages the rows.
//
// Products of a complex value and a real table entry are one packed
// fma.rn.f32x2 in FP32 (the FMA rate of two scalar ones at half the issue slots).
// FP64 is bound by the FP64 pipe (64 clocks per warp instruction on one of the
// four partitions of an SM); its tiles are one row / one latitude.  The sums run
// over latitudes (rows) in ascending order, one accumulator per term, whatever
// the tile: the results do not depend on the ensemble size.  Level chunks shrink
// for small ensembles until the units cover the SMs.
//
// k_anal is persistent and warp-specialised, one block per SM: consumer warps do
// nothing but the products while others fill the next stages; with every warp
// loading, folding and multiplying in turn it spent two thirds of its time
// between barriers.  Its waits on the stage barriers are bounded (tc_common.cuh):
// a role that gives up sets bit 1 of err and leaves, the others follow.
// k_synth, whose stores (as many bytes as HBM takes in that time) would stall the
// consumers, runs as plain blocks, two per SM, and was faster so (0.57 against
// 0.70 ms at 512 members).
#pragma once

namespace lbm {

// ---- packed complex accumulators --------------------------------------------
template <typename R> struct Cacc;
template <> struct Cacc<float> {
  unsigned long long v;
  using Fac = unsigned long long;     // a real factor in both halves
  static LBM_D Fac fac(float s) {
    Fac r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(s));
    return r;
  }
  LBM_D void zero() { v = 0ull; }
  LBM_D void fma(Fac s, unsigned long long x) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(s), "l"(x), "l"(v));
    v = r;
  }
  static LBM_D unsigned long long fma2(unsigned long long a, Fac s, unsigned long long b) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(s), "l"(b));
    return r;
  }
  LBM_D C2<float> get() const {
    C2<float> c;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(c.x), "=f"(c.y) : "l"(v));
    return c;
  }
};
template <> struct Cacc<double> {
  C2<double> v;
  using Fac = double;
  static LBM_D Fac fac(double s) { return s; }
  LBM_D void zero() { v = cmk<double>(0, 0); }
  LBM_D void fma(Fac s, C2<double> x) { cfma(v, s, x); }
  static LBM_D C2<double> fma2(C2<double> a, Fac s, C2<double> b) {
    cfma(b, s, a);
    return b;
  }
  LBM_D C2<double> get() const { return v; }
};
LBM_D void ld1(const C2<float>* p, unsigned long long& a) {
  a = *reinterpret_cast<const unsigned long long*>(p);
}
// One complex value in one shared-memory access (C2<float> itself is only
// 4-byte aligned); the address is a multiple of its size.
LBM_D C2<float> ldc(const C2<float>* p) {
  const float2 t = *reinterpret_cast<const float2*>(p);
  return cmk<float>(t.x, t.y);
}
LBM_D void stc(C2<float>* p, C2<float> a) { *reinterpret_cast<float2*>(p) = make_float2(a.x, a.y); }
LBM_D C2<double> ldc(const C2<double>* p) {
  const double2 t = *reinterpret_cast<const double2*>(p);
  return cmk<double>(t.x, t.y);
}
LBM_D void stc(C2<double>* p, C2<double> a) {
  *reinterpret_cast<double2*>(p) = make_double2(a.x, a.y);
}
LBM_D void ld1(const C2<double>* p, C2<double>& a) { a = ldc(p); }
// One complex value to global memory; nat: the address is a multiple of its size.
template <typename R> LBM_D void stg(C2<R>* p, C2<R> a, bool nat) {
  if (sizeof(R) == 4 && nat) stc(p, a);
  else *p = a;
}
template <typename R> struct Cval { using T = C2<double>; };
template <> struct Cval<float> { using T = unsigned long long; };

// A (P, H) table entry.  FP32 with DUP holds each value twice, ready as the factor
// of a packed product (making the pair in registers takes a move or two per
// factor); without it (tables that would not fit) it holds them once.
template <typename R, bool DUP> struct PH;
template <> struct alignas(16) PH<float, true> {
  float2 p, h;
  LBM_D void set(float P, float H) { p = make_float2(P, P); h = make_float2(H, H); }
  LBM_D float P() const { return p.x; }
};
template <> struct alignas(8) PH<float, false> {
  float p, h;
  LBM_D void set(float P, float H) { p = P; h = H; }
  LBM_D float P() const { return p; }
};
template <bool DUP> struct alignas(16) PH<double, DUP> {
  double p, h;
  LBM_D void set(double P, double H) { p = P; h = H; }
  LBM_D double P() const { return p; }
};
LBM_D void ldph(const PH<float, true>* t, unsigned long long& P, unsigned long long& H) {
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(t);
  P = v.x;
  H = v.y;
}
LBM_D void ldph(const PH<float, false>* t, unsigned long long& P, unsigned long long& H) {
  const float2 v = *reinterpret_cast<const float2*>(t);
  P = Cacc<float>::fac(v.x);
  H = Cacc<float>::fac(v.y);
}
template <bool DUP> LBM_D void ldph(const PH<double, DUP>* t, double& P, double& H) {
  const double2 v = *reinterpret_cast<const double2*>(t);
  P = v.x;
  H = v.y;
}

// ---- rows of an m-pair ----------------------------------------------------------
template <typename R> struct PairRows {
  int m1, m2, L1, L2, NR;
  LBM_HD PairRows(int p, int N) {
    m1 = p;
    m2 = N - p;
    L1 = N + 1 - m1;
    L2 = (m2 != m1) ? N + 1 - m2 : 0;
    NR = L1 + L2;
  }
  LBM_HD int m_of(int r) const { return r < L1 ? m1 : m2; }
  LBM_HD int n_of(int r) const { return r < L1 ? m1 + r : m2 + (r - L1); }
};

// Rows of an m-pair in table order: (m1, even), (m1, odd), (m2, even), (m2, odd)
// rows one list after the other, so that the rows of a group are adjacent and an
// odd row stride keeps adjacent groups apart in the shared-memory banks.
LBM_HD int table_pos(int r, int L1, int L2) {
  const int q = r < L1 ? r : r - L1, L = r < L1 ? L1 : L2;
  return (r < L1 ? 0 : L1) + ((q & 1) ? (L + 1) / 2 : 0) + q / 2;
}
// Groups of RT rows of one list.
template <int RT> struct PairGroups {
  int c[4];                           // rows of the lists
  LBM_HD PairGroups(int L1, int L2) {
    c[0] = (L1 + 1) / 2; c[1] = L1 / 2; c[2] = (L2 + 1) / 2; c[3] = L2 / 2;
  }
  LBM_HD int total() const {
    int t = 0;
    for (int l = 0; l < 4; ++l) t += (c[l] + RT - 1) / RT;
    return t;
  }
  // list of group x, its first table position, its rows and their first row in the m
  LBM_HD int list(int x, int* t0, int* n, int* r0) const {
    int l = 0, t = 0;
    while (l < 3 && x >= (c[l] + RT - 1) / RT) {
      x -= (c[l] + RT - 1) / RT;
      t += c[l++];
    }
    *t0 = t + RT * x;
    *n = c[l] - RT * x < RT ? c[l] - RT * x : RT;
    *r0 = (l & 1) + 2 * RT * x;
    return l;
  }
};

// Contiguous run of units of a persistent block.
LBM_D void unit_range(int units, int* u0, int* u1) {
  *u0 = (int)((long long)units * blockIdx.x / gridDim.x);
  *u1 = (int)((long long)units * (blockIdx.x + 1) / gridDim.x);
}
// Barrier of the consumer warps (id 1); true if any of them asks to stop.
LBM_D bool consumers_agree(int threads, bool stop) {
  unsigned any;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %2, 0;\n\t"
      "bar.red.or.pred q, 1, %1, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}\n"
      : "=r"(any)
      : "r"(threads), "r"((unsigned)stop)
      : "memory");
  return any != 0;
}
constexpr int LF_ERR = 2;             // bit of err set by a wait that gave up
// Barrier (id 2) after the first table is staged by the consumers and, where the
// consumers are few, by helper warps that do nothing else.
LBM_D void table_barrier(int threads) {
  asm volatile("bar.sync 2, %0;\n" ::"r"(threads) : "memory");
}
constexpr int LF_TABLE_WARPS = 8;     // warps that stage the first table

// Units in (pair, chunk, member) order, member fastest.
struct Unit {
  int u, p, z, e;
  LBM_D Unit(int u_, int nch, int E) : u(u_) {
    const int pz = u / E;
    e = u - pz * E;
    p = pz / nch;
    z = pz - p * nch;
  }
  LBM_D void next(int nch, int E) {
    ++u;
    if (++e == E) {
      e = 0;
      if (++z == nch) { z = 0; ++p; }
    }
  }
};

// Members per block of the surface-only kernels.
inline int members_per_block(int E, int units) {
  const int eb = (E * units) / (8 * FILL_SMS);
  return eb < 1 ? 1 : eb > 8 ? 8 : eb;
}

// =============================================================================
// Legendre analysis
// =============================================================================
struct AnalPlan {
  int KC, nch, G, CW, HW, JC, units, dup;   // levels per unit, chunks, row groups, consumer
                                      //   and helper warps, latitude pairs per stage, units,
                                      //   PH form
  int js, rst, oring;                 // strides of a table row and of a staged row, byte
                                      //   offset of the ring
  unsigned smem;
};
template <typename R> struct AnalCfg;
// rows of a tile, levels run over first by adjacent lanes
template <> struct AnalCfg<float> { static constexpr int RT = 3, LP = 2; };
template <> struct AnalCfg<double> { static constexpr int RT = 1, LP = 1; };
constexpr int AN_CW = 11;             // most consumer warps
constexpr int AN_FW = 5;              // warps that copy (FP64: and fold)
constexpr int AN_NV = 8;              // most vectors of a stage per copying thread
constexpr int AN_NS = 6, AN_DEPTH = 4;   // stages of the ring, and how many are being loaded
constexpr int AN_NT = 32 * (AN_CW + AN_FW);
static_assert(LF_TABLE_WARPS <= AN_CW, "helpers and consumers fit the block");

template <typename R> AnalPlan anal_plan(int E, int J, int K, int N) {
  using Cf = AnalCfg<R>;
  constexpr int RT = Cf::RT, LP = Cf::LP;
  const int JH = J / 2, NP = (N + 2) / 2, NR = N + 2;
  const int even = sizeof(R) == 4 && (K & 1) == 0;
  const size_t C = sizeof(C2<R>);
  AnalPlan p;
  p.G = 1;
  for (int q = 0; q < NP; ++q) {
    const PairRows<R> pr(q, N);
    const int g = PairGroups<RT>(pr.L1, pr.L2).total();
    if (g > p.G) p.G = g;
  }
  p.js = JH | 1;
  p.HW = 0;
  // chunks of the levels (the surface is one more level of the last chunk): as
  // few as AN_CW warps hold; more for small ensembles, down to four levels, while
  // units do not outnumber the SMs
  int nch = 1;
  while (nch < (K + 3) / 4 && NP * E * (nch + 1) <= FILL_SMS) ++nch;
  for (;; ++nch) {
    p.KC = (K + nch - 1) / nch;
    if (even) p.KC += p.KC & 1;
    p.nch = (K + p.KC - 1) / p.KC;
    const int last = K - (p.nch - 1) * p.KC + 1, most = last > p.KC ? last : p.KC;
    p.CW = ((most + LP - 1) / LP * LP * p.G + 31) / 32;
    p.units = NP * E * p.nch;
    // row and surface values; the rows of the four (m, parity) are 16 bytes apart
    // (mod 128) in the banks
    p.rst = p.KC * AF_N + 2;
    while (sizeof(R) == 4 ? (p.rst % 16 != 2 && p.rst % 16 != 14) : (p.rst % 8 != 1 && p.rst % 8 != 7))
      ++p.rst;
    for (p.dup = sizeof(R) == 4;; p.dup = 0) {
      // (a group may read up to RT - 1 rows past the table)
      const size_t ent = p.dup || sizeof(R) == 8 ? 16 : 8;
      p.oring = (int)((128 + ent * (NR + RT - 1) * (size_t)p.js + 15) & ~size_t(15));
      const int most_jc = AN_NV * 32 * AN_FW * (even ? 2 : 1) / (2 * AF_N * p.KC);
      p.JC = 18432 / (int)(C * 4 * p.rst);                   // about 18 KB per stage
      if (p.JC > most_jc) p.JC = most_jc;
      if (p.JC > 8 * AN_FW) p.JC = 8 * AN_FW;                // one surface value per thread
      if (p.JC > JH) p.JC = JH;
      if (p.JC < 1) p.JC = 1;
      for (;; --p.JC) {
        // (a surface item reads up to AF_N values from the end of a row)
        p.smem = (unsigned)(p.oring + C * (AN_NS * (size_t)p.JC * 4 * p.rst + AF_N));
        if (p.smem <= 227 * 1024 || p.JC == 1) break;
      }
      if (p.smem <= 227 * 1024 || !p.dup) break;
    }
    if ((p.smem <= 227 * 1024 && p.CW <= AN_CW) || p.KC <= 1 + even) break;
  }
  if (p.CW < LF_TABLE_WARPS) p.HW = LF_TABLE_WARPS - p.CW;
  return p;
}

// (P, H) of the pair's rows in table order, [NR][js], by nw warps, this one w0.
template <typename R, bool DUP>
LBM_D void anal_table(const SD<R>& d, const PairRows<R>& pr, PH<R, DUP>* tab, int js, int w0,
                      int nw) {
  const int JH = d.J / 2, off1 = spec_offset(pr.m1, d.N), off2 = spec_offset(pr.m2, d.N);
  const int lane = threadIdx.x & 31;
#pragma unroll 2
  for (int r = w0; r < pr.NR; r += nw) {
    const size_t o = (size_t)(r < pr.L1 ? off1 + r : off2 + (r - pr.L1)) * JH;
    PH<R, DUP>* t = tab + table_pos(r, pr.L1, pr.L2) * js;
    for (int jh = lane; jh < JH; jh += 32) t[jh].set(d.symp[o + jh], d.symh[o + jh]);
  }
}

// Surface rows (gt_pi, pi(t - dt)) of members e0 .. e1 - 1: one thread per
// (row, field); xs: room for 8 JH values.
template <typename R>
LBM_D void anal_surface(const SD<R>& d, int p, int e0, int e1, const PH<R, false>* tab, int js,
                        C2<R>* xs) {
  const int J = d.J, N = d.N, M = d.M, JH = J / 2;           // xs [2 m][JH][2 fields][2 parities]
  const PairRows<R> pr(p, N);
  const int tid = threadIdx.x, nt = blockDim.x;
  const FastDiv fjh(JH);
  const int nm = pr.L2 ? 2 : 1;
  for (int e = e0; e < e1; ++e) {
    __syncthreads();
    for (int x = tid; x < nm * JH * 2; x += nt) {
      const int f = x & 1, q = x >> 1, mm = fjh.div(q), jh = q - mm * JH;
      const int m = mm ? pr.m2 : pr.m1;
      const C2<R>* a = d.afs + ((size_t)e * M + m) * J * 2 + f;
      const C2<R> xn = a[2 * jh], xsouth = a[2 * (J - 1 - jh)];
      stc(xs + (q * 2 + f) * 2, xn + xsouth);
      stc(xs + (q * 2 + f) * 2 + 1, xn - xsouth);
    }
    __syncthreads();
    for (int x = tid; x < pr.NR * 2; x += nt) {
      const int f = x >= pr.NR, r = x - f * pr.NR;
      const int mm = r < pr.L1 ? 0 : 1, m = pr.m_of(r), n = pr.n_of(r);
      const C2<R>* s = xs + (mm * JH * 2 + f) * 2 + ((n - m) & 1);
      const PH<R, false>* t = tab + table_pos(r, pr.L1, pr.L2) * js;
      C2<R> a = cmk<R>(0, 0);
#pragma unroll 4
      for (int jh = 0; jh < JH; ++jh) cfma(a, t[jh].P(), ldc(s + jh * 4));
      d.tends[((size_t)e * 2 + f) * d.NS + spec_index(m, n, N)] = a;
    }
  }
}

LBM_HD size_t anal_surf_smem(int J, int N) {
  return 8 * (N + 2) * (size_t)((J / 2) | 1) + 8 + sizeof(C2<float>) * 4 * (size_t)J;
}
__global__ void __launch_bounds__(128) k_anal_surf(SD<float> d, int eb) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const PairRows<float> pr(blockIdx.x, d.N);
  const int js = (d.J / 2) | 1, e0 = blockIdx.y * eb;
  PH<float, false>* tab = reinterpret_cast<PH<float, false>*>(smraw);
  anal_table(d, pr, tab, js, threadIdx.x >> 5, 4);
  anal_surface(d, blockIdx.x, e0, min(d.E, e0 + eb), tab, js,
               reinterpret_cast<C2<float>*>(tab + (d.N + 2) * js));
}

// Unit: (m-pair, level chunk, member); the two surface fields are one more level
// of the last chunk (P sums only).  The northern and southern rows of JC latitude
// pairs stream into a ring of AN_NS stages.  A consumer thread owns RT rows of one
// parity at one level, nine sums each (P: FU FV KE T Q of the row's parity, H: FU
// FV XV YV of the other).  Its items run over two levels first (lane pairs share
// the 16-byte table entries), then over the row groups (lanes share a level's
// values).  Sums go straight to global memory.
// Five warps copy the rows with cp.async, AN_DEPTH stages ahead.  FP32 adds north
// and south in the consumers' registers (9 of 36 packed operations); warps that
// folded the rows in shared memory could not keep up, nor could one warp of bulk
// copies (1 KB each, some 40 ns).  FP64, bound by its pipe, folds in the copying
// warps, each thread the vectors it copied.
// us at T42L20 against the block-per-(pair, member) kernel before: FP32 11 (26), 189
// (264), 720 (1009) at 1, 128, 512 members; T85L40, 16 members 335 (444); FP64 41
// (149), 720 (1329) at 1, 32 members, the FP64 pipe's time for the products 670.
template <typename R, int VEC, bool DUP>
__global__ void __launch_bounds__(AN_NT, 1) k_anal(SD<R> d, AnalPlan pl) {
  constexpr bool FOLD = sizeof(R) == 8;
  constexpr int FW = AN_FW;
  constexpr int RT = AnalCfg<R>::RT, LP = AnalCfg<R>::LP;
  using V = typename Cval<R>::T;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int J = d.J, K = d.K, N = d.N, M = d.M, E = d.E, JH = J / 2;
  const int JC = pl.JC, JS = pl.js, rst = pl.rst, CW = pl.CW, nch = pl.nch;
  const unsigned bfull = tc::smem_addr(smraw), bempty = bfull + 8 * AN_NS;
  PH<R, DUP>* tab = reinterpret_cast<PH<R, DUP>*>(smraw + 128);   // [NR][JS]
  C2<R>* ring = reinterpret_cast<C2<R>*>(smraw + pl.oring);   // [AN_NS][JC][2 m][2 par][rst]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int bsz = JC * 4 * rst, nst = (JH + JC - 1) / JC;
  if (tid == 0) {
    for (int i = 0; i < AN_NS; ++i) {
      tc::mbar_init(bfull + 8 * i, FW);
      tc::mbar_init(bempty + 8 * i, CW);
    }
    tc::fence_mbar_init();
  }
  __syncthreads();
  int u0, u1;
  unit_range(pl.units, &u0, &u1);
  bool ok = true;
  if (warp < CW || warp >= CW + FW) {
    // the first table, with the helper warps
    const Unit un(u0, nch, E);
    anal_table(d, PairRows<R>(un.p, N), tab, JS, warp < CW ? warp : warp - FW, CW + pl.HW);
    table_barrier(32 * (CW + pl.HW));
  }
  if (warp < CW) {
    // ---------------- consumers ----------------
    int s = 0, cur = u0 / (nch * E);
    unsigned ph = 0;
    const bool nat = ((uintptr_t)d.tend & (sizeof(C2<R>) - 1)) == 0;
    for (Unit un(u0, nch, E); un.u < u1; un.next(nch, E)) {
      const int e = un.e, p = un.p, z = un.z;
      const PairRows<R> pr(p, N);
      // all are done with the previous unit (and its table)
      if (consumers_agree(32 * CW, !ok)) break;
      if (p != cur) {
        anal_table(d, pr, tab, JS, warp, CW);
        consumers_agree(32 * CW, false);
        cur = p;
      }
      const int k0 = z * pl.KC, kn = min(pl.KC, K - k0), surf = z == nch - 1;
      const PairGroups<RT> pg(pr.L1, pr.L2);
      const int G = pg.total();
      const int it = tid / LP, kp = it / G, g = it - kp * G, k = LP * kp + (tid & (LP - 1));
      const bool active = k < kn + surf;
      int t0, cnt, r0;
      const int li = pg.list(g, &t0, &cnt, &r0), mi = li >> 1, par = li & 1;
      // folded rows: the row's parity for P, the other for H; else north and south
      const int xo = (2 * mi + (FOLD ? par : 0)) * rst + k * AF_N;
      const int ho = (2 * mi + (FOLD ? par ^ 1 : 1)) * rst + k * AF_N;
      const auto sgp = Cacc<R>::fac(par ? R(-1) : R(1)), sgh = Cacc<R>::fac(par ? R(1) : R(-1));
      Cacc<R> acc[RT][9];
#pragma unroll
      for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int a = 0; a < 9; ++a) acc[i][a].zero();
      const PH<R, DUP>* tb = tab + t0 * JS;
      for (int jh0 = 0; jh0 < JH; jh0 += JC) {
        ok = ok && tc::warp_wait(bfull + 8 * s, ph, d.err, LF_ERR);
        if (!ok) break;
        const C2<R> *xp = ring + s * bsz + xo, *xh = ring + s * bsz + ho;
        const int jc = min(JC, JH - jh0);
        if (active) {
#pragma unroll 4
          for (int jj = 0; jj < jc; ++jj, xp += 4 * rst, xh += 4 * rst, ++tb) {
            V fu, fv, ke, t, q, hu, hv, xv, yv;
            ld1(xp + AF_FU, fu);
            ld1(xp + AF_FV, fv);
            ld1(xp + AF_KE, ke);
            ld1(xp + AF_T, t);
            ld1(xp + AF_Q, q);
            ld1(xh + AF_FU, hu);
            ld1(xh + AF_FV, hv);
            ld1(xh + AF_XV, xv);
            ld1(xh + AF_YV, yv);
            if constexpr (!FOLD) {
              // north +- south (times +-1: exact)
              V ke2, t2, q2, xv2, yv2;
              ld1(xh + AF_KE, ke2);
              ld1(xh + AF_T, t2);
              ld1(xh + AF_Q, q2);
              ld1(xp + AF_XV, xv2);
              ld1(xp + AF_YV, yv2);
              const V fun = fu, fvn = fv;
              fu = Cacc<R>::fma2(hu, sgp, fun);
              fv = Cacc<R>::fma2(hv, sgp, fvn);
              ke = Cacc<R>::fma2(ke2, sgp, ke);
              t = Cacc<R>::fma2(t2, sgp, t);
              q = Cacc<R>::fma2(q2, sgp, q);
              hu = Cacc<R>::fma2(hu, sgh, fun);
              hv = Cacc<R>::fma2(hv, sgh, fvn);
              xv = Cacc<R>::fma2(xv, sgh, xv2);
              yv = Cacc<R>::fma2(yv, sgh, yv2);
            }
#pragma unroll
            for (int i = 0; i < RT; ++i) {
              typename Cacc<R>::Fac P, H;
              ldph(tb + i * JS, P, H);
              acc[i][0].fma(P, fu);
              acc[i][1].fma(P, fv);
              acc[i][2].fma(P, ke);
              acc[i][3].fma(P, t);
              acc[i][4].fma(P, q);
              acc[i][5].fma(H, hu);
              acc[i][6].fma(H, hv);
              acc[i][7].fma(H, xv);
              acc[i][8].fma(H, yv);
            }
          }
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(bempty + 8 * s);
        if (++s == AN_NS) { s = 0; ph ^= 1u; }
      }
      if (!ok) continue;
      if (active) {
        const int m = mi ? pr.m2 : pr.m1, row = spec_offset(m, N) + r0;
        const R rm = R(m);
        const size_t SO = (size_t)d.NS * K;
        C2<R>* te = d.tend + (size_t)e * 4 * SO + (size_t)row * K + k0 + k;
#pragma unroll
        for (int i = 0; i < RT; ++i) {
          if (i >= cnt) break;
          if (k < kn) {
            C2<R>* o = te + 2 * i * K;
            stg(o, im_mul(acc[i][1].get(), rm) + acc[i][5].get(), nat);
            stg(o + SO, im_mul(acc[i][0].get(), rm) - acc[i][6].get() +
                            acc[i][2].get() * d.nn1a[m + r0 + 2 * i], nat);
            stg(o + 2 * SO, acc[i][3].get() + acc[i][7].get(), nat);
            stg(o + 3 * SO, acc[i][4].get() + acc[i][8].get(), nat);
          } else {
            C2<R>* o = d.tends + (size_t)e * 2 * d.NS + row + 2 * i;
            o[0] = acc[i][0].get();
            o[d.NS] = acc[i][1].get();
          }
        }
      }
    }
  } else {
    // ---------------- copy (FP64: and fold) ----------------
    if (warp >= CW + FW) return;
    const int ft = tid - 32 * CW;
    constexpr int FT = 32 * AN_FW;
    const int jK = K * AF_N;
    const int T = (u1 - u0) * nst;
    // Stage t is copied at step t and folded at step t + AN_DEPTH.  This thread's
    // vectors of a stage, for the (pair, chunk) of the stage being copied: source
    // offset within the latitude rows, latitude pair in the stage (-1: none), place
    // in the slot.  A vector of the surface fields is one value.
    struct Mine {
      int o[AN_NV], src[AN_NV], jj[AN_NV], so, sj, ssrc, key;
    };
    auto place = [&](Mine& v, const Unit& un) {
      if (v.key == un.p * nch + un.z) return;
      v.key = un.p * nch + un.z;
      const PairRows<R> pr(un.p, N);
      const int k0 = un.z * pl.KC, kn = min(pl.KC, K - k0), nm = pr.L2 ? 2 : 1;
      const int nv = kn * AF_N / VEC;
      const FastDiv fv(nv);
#pragma unroll
      for (int i = 0; i < AN_NV; ++i) {
        const int x = ft + i * FT, w = fv.div(x), c = (x - w * nv) * VEC;
        const int jj = nm == 2 ? w >> 1 : w, mm = nm == 2 ? w & 1 : 0;
        v.jj[i] = jj < JC ? jj : JH;
        v.o[i] = (4 * jj + 2 * mm) * rst + c;
        v.src[i] = (mm ? pr.m2 : pr.m1) * J * jK + k0 * AF_N + c;
      }
      // surface: value f of pair w at x = 2 w + f
      const int w = ft >> 1, f = ft & 1, jj = nm == 2 ? w >> 1 : w, mm = nm == 2 ? w & 1 : 0;
      v.sj = un.z == nch - 1 && jj < JC ? jj : JH;
      v.so = (4 * jj + 2 * mm) * rst + kn * AF_N + f;
      v.ssrc = ((mm ? pr.m2 : pr.m1) * J) * 2 + f;
    };
    Unit ui(u0, nch, E), uf(u0, nch, E);
    // (afs may lie off its element's alignment, which cp.async does not take)
    const bool nats = ((uintptr_t)d.afs & (sizeof(C2<R>) - 1)) == 0;
    Mine vi, vf;
    vi.key = vf.key = -1;
    int ji = 0, jf = 0, si = 0, sf = 0;
    unsigned ph = 0;
    for (int t = 0; t < T + AN_DEPTH; ++t) {
      if (t < T) {
        if (!tc::warp_wait(bempty + 8 * si, ph ^ 1u, d.err, LF_ERR)) break;
        place(vi, ui);
        const C2<R>* src = d.af + (size_t)ui.e * M * J * jK;
        C2<R>* dst = ring + si * bsz;
        const int left = JH - ji;
#pragma unroll
        for (int i = 0; i < AN_NV; ++i)
          if (vi.jj[i] < left) {
            const int jn = ji + vi.jj[i];
            const C2<R>* a = src + vi.src[i];
            C2<R>* o = dst + vi.o[i];
            if constexpr (VEC == 2) {
              cp_async16(o, a + jn * jK);
              cp_async16(o + rst, a + (J - 1 - jn) * jK);
            } else {
              cp_async_c2(o, a + jn * jK);
              cp_async_c2(o + rst, a + (J - 1 - jn) * jK);
            }
          }
        if (vi.sj < left) {
          const C2<R>* a = d.afs + (size_t)ui.e * M * J * 2 + vi.ssrc;
          const C2<R>*n1 = a + 2 * (ji + vi.sj), *s1 = a + 2 * (J - 1 - ji - vi.sj);
          C2<R>* o = dst + vi.so;
          if (nats) {
            cp_async_c2(o, n1);
            cp_async_c2(o + rst, s1);
          } else {
            o[0] = *n1;
            o[rst] = *s1;
          }
        }
        ji += JC;
        if (ji >= JH) { ji = 0; ui.next(nch, E); }
        if (++si == AN_NS) { si = 0; ph ^= 1u; }
      }
      cp_async_commit();
      if (t >= AN_DEPTH) {
        cp_async_wait<AN_DEPTH>();
        place(vf, uf);
        C2<R>* dst = ring + sf * bsz;
        const int left = JH - jf;
        if constexpr (FOLD) {
#pragma unroll
          for (int i = 0; i < AN_NV; ++i)
            if (vf.jj[i] < left) {
              C2<R>* o = dst + vf.o[i];
              const C2<R> n1 = ldc(o), s1 = ldc(o + rst);
              stc(o, n1 + s1);
              stc(o + rst, n1 - s1);
            }
          if (vf.sj < left) {
            C2<R>* o = dst + vf.so;
            const C2<R> n1 = ldc(o), s1 = ldc(o + rst);
            stc(o, n1 + s1);
            stc(o + rst, n1 - s1);
          }
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(bfull + 8 * sf);
        jf += JC;
        if (jf >= JH) { jf = 0; uf.next(nch, E); }
        if (++sf == AN_NS) sf = 0;
      }
    }
    cp_async_wait<0>();
  }
}

template <typename R> void launch_anal(const SD<R>& d, cudaStream_t st, bool attrs) {
  const AnalPlan pl = anal_plan<R>(d.E, d.J, d.K, d.N);
  auto go = [&](auto kern) {
    if (attrs) {
      allow_smem(kern);
    } else {
      const int sms = device_sms();
      kern<<<pl.units < sms ? pl.units : sms, 32 * (pl.CW + pl.HW + AN_FW), pl.smem, st>>>(d, pl);
    }
  };
  // 16-byte copies: FP32 rows of an even level count (and always in FP64)
  if constexpr (sizeof(R) == 8) {
    go(k_anal<R, 1, true>);
  } else if (pl.dup) {
    if (d.K & 1) go(k_anal<R, 1, true>);
    else go(k_anal<R, 2, true>);
  } else {
    if (d.K & 1) go(k_anal<R, 1, false>);
    else go(k_anal<R, 2, false>);
  }
}

// =============================================================================
// Legendre synthesis
// =============================================================================
struct SynthPlan {
  int NJG, NJQ, QC, nch, nt, eb;      // latitude groups, quads of them, level quads per block,
                                      //   chunks, threads, members per block
  int jhp, ntab, bufs, oil, ox;       // table row stride, tables, state buffers, byte offsets
                                      //   of the inverse Laplacian factors and of the state
  unsigned smem;
};
template <typename R> struct SynthCfg;
// FP64 folds the inverse Laplacian factor into the tables (P, P il, H il) instead
// of scaling each coefficient: four of twenty FP64 operations per row less.  Where
// the third table leaves no room for a level quad of one member ((nmax + 2)
// (nlat / 2 + 11) above 9,685) there are two, as in FP32: by the grid alone, so that
// a member's results do not depend on the ensemble.
template <> struct SynthCfg<float> { static constexpr int JG = 4, NW = 10, NTAB = 2; };
template <> struct SynthCfg<double> { static constexpr int JG = 1, NW = 8, NTAB = 3; };

template <typename R> SynthPlan synth_plan(int E, int J, int K, int N) {
  constexpr int JG = SynthCfg<R>::JG, NW = SynthCfg<R>::NW;
  const int JH = J / 2, NP = (N + 2) / 2, nq = (K + 3) / 4;
  const size_t NR = N + 2, C = sizeof(C2<R>);
  SynthPlan p;
  p.NJG = (JH + JG - 1) / JG;
  p.NJQ = (p.NJG + 3) / 4;
  p.jhp = p.NJG * JG;
  // level quads per block: one warp per (latitude, level) quad up to NW (FP64:
  // three rounds, so that fewer blocks stage the tables), but blocks for two per
  // SM
  int qc = (sizeof(R) == 4 ? 1 : 3) * NW / p.NJQ;
  if (qc < 1) qc = 1;
  int nch = (nq + qc - 1) / qc;
  int want = (2 * FILL_SMS + NP * E - 1) / (NP * E);
  if (want > nq) want = nq;
  if (nch < want) nch = want;
  auto layout = [&](int ntab, int qc_, int bufs) {
    const int kc = 4 * qc_ < K ? 4 * qc_ : K;
    p.ntab = ntab;
    p.bufs = bufs;
    p.oil = (int)((sizeof(R) * ntab * NR * (size_t)p.jhp + 15) & ~size_t(15));
    p.ox = (int)((p.oil + sizeof(R) * NR + 15) & ~size_t(15));
    size_t x = bufs * C * NR * 4 * (size_t)kc;
    if (x < C * NR * 4) x = C * NR * 4;                      // the surface fields
    p.smem = (unsigned)(p.ox + x);
    return p.smem;
  };
  const int ntab = layout(SynthCfg<R>::NTAB, 1, 1) <= 227 * 1024 ? SynthCfg<R>::NTAB : 2;
  for (;; ++nch) {
    p.QC = (nq + nch - 1) / nch;
    p.nch = (nq + p.QC - 1) / p.QC;
    p.eb = members_per_block(E, NP * p.nch);
    if (layout(ntab, p.QC, p.eb > 1 ? 2 : 1) <= 113 * 1024 || p.QC == 1) break;
  }
  // one member a block where two buffers do not fit
  if (p.smem > 227 * 1024) {
    p.eb = 1;
    layout(ntab, p.QC, 1);
  }
  const int w = p.NJQ * p.QC;
  p.nt = 32 * (w < NW ? w : NW);
  if (NP * E * p.nch <= 2 * FILL_SMS && p.nt < 192) p.nt = 192;   // threads to stage with
  if (p.nt < 64) p.nt = 64;
  return p;
}

// Tables of the pair's rows, [NR][JHp], zero past the equator: P and H, or P, P il
// and H il.
template <typename R, int NTAB>
LBM_D void synth_tables(const SD<R>& d, const PairRows<R>& pr, R* tp, int JHp) {
  const int JH = d.J / 2, off1 = spec_offset(pr.m1, d.N), off2 = spec_offset(pr.m2, d.N);
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5, TT = (d.N + 2) * JHp;
#pragma unroll 2
  for (int r = threadIdx.x >> 5; r < pr.NR; r += nw) {
    const size_t o = (size_t)(r < pr.L1 ? off1 + r : off2 + (r - pr.L1)) * JH;
    const R il = NTAB == 3 ? d.invlap[pr.n_of(r)] : R(1);
    for (int jh = lane; jh < JHp; jh += 32) {
      const R P = jh < JH ? d.symp[o + jh] : R(0), H = jh < JH ? d.symh[o + jh] : R(0);
      R* t = tp + r * JHp + jh;
      t[0] = P;
      if constexpr (NTAB == 3) {
        t[TT] = P * il;
        t[2 * TT] = H * il;
      } else {
        t[TT] = H;
      }
    }
  }
}

// Surface fields (pi, H pi, column-sum winds and divergence) of members e0 ..
// e1 - 1: one thread per (m, latitude pair), the coefficients staged in xs.
template <typename R>
LBM_D void synth_surface(const SD<R>& d, int p, int e0, int e1, const R* tp, const R* th, int jhp,
                         C2<R>* xs) {
  const int J = d.J, N = d.N, M = d.M, JH = J / 2, NS = d.NS;
  const PairRows<R> pr(p, N);
  const int tid = threadIdx.x, nt = blockDim.x;
  const int off1 = spec_offset(pr.m1, N), off2 = spec_offset(pr.m2, N);
  const int nm = pr.L2 ? 2 : 1;
  const FastDiv fr(pr.NR);
  for (int e = e0; e < e1; ++e) {
    __syncthreads();
    for (int x = tid; x < pr.NR * 4; x += nt) {
      const int f = fr.div(x), r = x - f * pr.NR;
      stc(xs + r * 4 + f,
          d.sas[((size_t)e * 4 + f) * NS + (r < pr.L1 ? off1 + r : off2 + (r - pr.L1))]);
    }
    __syncthreads();
    for (int it = tid; it < nm * JH; it += nt) {
      const int mm = it >= JH, jh = it - mm * JH;
      const int m = mm ? pr.m2 : pr.m1;
      const int rb = mm ? pr.L1 : 0, re = mm ? pr.NR : pr.L1;
      // terms: Ppi Hpi Pchis Hpsis Ppsis Hchis Pds  [plus/minus]
      C2<R> acc[7][2];
#pragma unroll
      for (int b = 0; b < 7; ++b) acc[b][0] = acc[b][1] = cmk<R>(0, 0);
      auto row = [&](int r, auto par_tag) {
        constexpr int PP = decltype(par_tag)::value, HP = PP ^ 1;
        const C2<R> pi = ldc(xs + r * 4), psis = ldc(xs + r * 4 + 1);
        const C2<R> chis = ldc(xs + r * 4 + 2), ds = ldc(xs + r * 4 + 3);
        const R P = tp[r * jhp + jh], H = th[r * jhp + jh];
        cfma(acc[0][PP], P, pi);
        cfma(acc[1][HP], H, pi);
        cfma(acc[2][PP], P, chis);
        cfma(acc[3][HP], H, psis);
        cfma(acc[4][PP], P, psis);
        cfma(acc[5][HP], H, chis);
        cfma(acc[6][PP], P, ds);
      };
      for (int r = rb; r < re; r += 2) {
        row(r, std::integral_constant<int, 0>{});
        if (r + 1 < re) row(r + 1, std::integral_constant<int, 1>{});
      }
      const R rm = R(m);
      for (int hemi = 0; hemi < 2; ++hemi) {
        const int j = hemi ? J - 1 - jh : jh;
        const R sg = hemi ? R(-1) : R(1);
        auto comb = [&](int b) { return acc[b][0] + acc[b][1] * sg; };
        C2<R>* o = d.sfs + (((size_t)e * M + m) * J + j) * SFS_N;
        o[SFS_PI] = comb(0);
        o[SFS_PIY] = comb(1);
        o[SFS_UH] = im_mul(comb(2), rm) - comb(3);
        o[SFS_VH] = im_mul(comb(4), rm) + comb(5);
        o[SFS_DH] = comb(6);
      }
    }
  }
}

__global__ void __launch_bounds__(128) k_synth_surf(SD<float> d, SynthPlan pl, int eb) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const PairRows<float> pr(blockIdx.x, d.N);
  const int e0 = blockIdx.y * eb;
  float* tp = reinterpret_cast<float*>(smraw);
  synth_tables<float, 2>(d, pr, tp, pl.jhp);
  synth_surface(d, blockIdx.x, e0, min(d.E, e0 + eb), tp, tp + (d.N + 2) * pl.jhp, pl.jhp,
                reinterpret_cast<C2<float>*>(smraw + pl.ox));
}

// Two adjacent complex values in one store (16 bytes in FP32; the six-field
// rows of sf start on 16-byte boundaries).
LBM_D void store_pair(C2<float>* o, C2<float> a, C2<float> b) {
  *reinterpret_cast<float4*>(o) = make_float4(a.x, a.y, b.x, b.y);
}
LBM_D void store_pair(C2<double>* o, C2<double> a, C2<double> b) {
  o[0] = a;
  o[1] = b;
}
template <typename R> LBM_D C2<R> shfl_xor_c(C2<R> a, int x) {
  return cmk<R>(__shfl_xor_sync(0xffffffffu, a.x, x), __shfl_xor_sync(0xffffffffu, a.y, x));
}
// x il, as the reference scales vorticity and divergence into psi and chi
LBM_D unsigned long long scale_c(unsigned long long x, unsigned long long il) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(il));
  return r;
}
LBM_D C2<double> scale_c(C2<double> x, double il) { return x * il; }

// Block (m-pair, eb members, chunk of QC level quads); chunk index 0 is the
// surface block.  A member's rows are staged as they lie in the state
// ([row][field][level], the next member's copies in flight).  A warp takes four
// levels x four latitude groups x the two row parities (lane bits 0-1, 2-3, 4:
// adjacent lanes share the 16-byte table loads); a thread accumulates the eight terms P chi, H psi, P psi, H chi (winds), P
// vor, P div, P T, P q of its rows at JG latitudes.
// us at T42L20 against one thread item for both parities before: FP32 11 (21), 159
// (208), 573 (784) at 1, 128, 512 members; T85L40, 16 members 225 (383); FP64 41
// (98), 682 (641) at 1, 32 members.
template <typename R, int MINB, int NTAB>
__global__ void __launch_bounds__(32 * SynthCfg<R>::NW, MINB) k_synth(SD<R> d, SynthPlan pl) {
  constexpr int JG = SynthCfg<R>::JG;
  using V = typename Cval<R>::T;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int p = blockIdx.x, e0 = blockIdx.y * pl.eb, e1 = min(d.E, e0 + pl.eb);
  const int J = d.J, K = d.K, N = d.N, M = d.M, JH = J / 2, NS = d.NS, JHp = pl.jhp;
  const PairRows<R> pr(p, N);
  const int TT = (N + 2) * JHp;
  R* tp = reinterpret_cast<R*>(smraw);                       // [NTAB][NR][JHp]
  C2<R>* buf = reinterpret_cast<C2<R>*>(smraw + pl.ox);      // [bufs][NR][4][kn]
  if (blockIdx.z == 0) {                                     // first, so that no tail is left
    synth_tables<R, 2>(d, pr, tp, JHp);
    synth_surface(d, p, e0, e1, tp, tp + TT, JHp, buf);
    return;
  }
  R* ils = reinterpret_cast<R*>(smraw + pl.oil);             // inverse Laplacian of row r
  const int k0 = ((int)blockIdx.z - 1) * 4 * pl.QC, kn = min(4 * pl.QC, K - k0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  const int off1 = spec_offset(pr.m1, N), off2 = spec_offset(pr.m2, N);
  const size_t bsz = (size_t)pr.NR * 4 * kn;
  // 16-byte copies where the state and every row piece are so aligned, else one
  // value at a time (natural alignment), else plain loads
  const bool w16 = sizeof(R) == 8 ? ((uintptr_t)d.sa3 & 15) == 0
                                  : (((uintptr_t)d.sa3 & 15) == 0 && !(K & 1) && !(kn & 1));
  const bool w8 = sizeof(R) == 4 && ((uintptr_t)d.sa3 & 7) == 0;
  auto issue = [&](int e, C2<R>* b) {
    const C2<R>* st = d.sa3 + (size_t)e * 4 * NS * K + k0;
    constexpr int PER = 16 / (int)sizeof(C2<R>);
    const int nv = w16 ? kn / PER : kn;
    const FastDiv fv(nv);
    for (int x = tid; x < pr.NR * 4 * nv; x += blockDim.x) {
      const int y = fv.div(x), c = x - y * nv, r = y >> 2, f = y & 3;
      const C2<R>* src =
          st + ((size_t)f * NS + (r < pr.L1 ? off1 + r : off2 + (r - pr.L1))) * K;
      C2<R>* dst = b + (size_t)y * kn;
      if (w16) cp_async16(dst + c * PER, src + c * PER);
      else if (w8) cp_async_c2(dst + c, src + c);
      else dst[c] = src[c];
    }
    cp_async_commit();
  };
  issue(e0, buf);
  synth_tables<R, NTAB>(d, pr, tp, JHp);
  for (int r = tid; r < pr.NR; r += blockDim.x) ils[r] = d.invlap[pr.n_of(r)];
  const int par = lane >> 4, nm = pr.L2 ? 2 : 1, nq = (kn + 3) / 4;
  const R sg = par ? R(-1) : R(1);
  const size_t jmK = (size_t)J * K;
  int b = 0;
  for (int e = e0; e < e1; ++e, b ^= 1) {
    if (e + 1 < e1) {
      __syncthreads();                                       // the other buffer is read
      issue(e + 1, buf + (b ^ 1) * bsz);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const C2<R>* X = buf + b * bsz;
    C2<R>* sfe = d.sf + (size_t)e * M * jmK * SF_N;
    for (int w = warp; w < pl.NJQ * nq; w += nw) {
      const int kq = w / pl.NJQ, jq = w - kq * pl.NJQ;
      const int jg = 4 * jq + ((lane >> 2) & 3), kk = 4 * kq + (lane & 3);
      const bool live = jg < pl.NJG && kk < kn;
      const int jgc = min(jg, pl.NJG - 1), kc = min(kk, kn - 1);
      for (int mm = 0; mm < nm; ++mm) {
        const int m = mm ? pr.m2 : pr.m1;
        const int rb = mm ? pr.L1 : 0, re = mm ? pr.NR : pr.L1;
        const R rm = R(m);
        Cacc<R> acc[JG][8];
#pragma unroll
        for (int a = 0; a < JG; ++a)
#pragma unroll
          for (int q = 0; q < 8; ++q) acc[a][q].zero();
        const C2<R>* s = X + (rb + par) * 4 * kn + kc;
        const R* pp = tp + (rb + par) * JHp + jgc * JG;
        for (int r = rb + par; r < re; r += 2, s += 8 * kn, pp += 2 * JHp) {
          V vo, dv, tt, qq;
          ld1(s, vo);
          ld1(s + kn, dv);
          ld1(s + 2 * kn, tt);
          ld1(s + 3 * kn, qq);
          if constexpr (NTAB == 2 && JG == 1) {
            const R P = pp[0], H = pp[TT], il = ils[r];
            const V psi = scale_c(vo, il), chi = scale_c(dv, il);
            acc[0][0].fma(P, chi);
            acc[0][1].fma(H, psi);
            acc[0][2].fma(P, psi);
            acc[0][3].fma(H, chi);
            acc[0][4].fma(P, vo);
            acc[0][5].fma(P, dv);
            acc[0][6].fma(P, tt);
            acc[0][7].fma(P, qq);
          } else if constexpr (NTAB == 2) {
            const auto il = Cacc<R>::fac(ils[r]);
            const V psi = scale_c(vo, il), chi = scale_c(dv, il);
            const float4 u = *reinterpret_cast<const float4*>(pp);
            const float4 v = *reinterpret_cast<const float4*>(pp + TT);
            const float P[4] = {u.x, u.y, u.z, u.w}, H[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int a = 0; a < JG; ++a) {
              const auto Pf = Cacc<R>::fac(P[a]), Hf = Cacc<R>::fac(H[a]);
              acc[a][0].fma(Pf, chi);
              acc[a][1].fma(Hf, psi);
              acc[a][2].fma(Pf, psi);
              acc[a][3].fma(Hf, chi);
              acc[a][4].fma(Pf, vo);
              acc[a][5].fma(Pf, dv);
              acc[a][6].fma(Pf, tt);
              acc[a][7].fma(Pf, qq);
            }
          } else {
#pragma unroll
            for (int a = 0; a < JG; ++a) {
              const R P = pp[a], Pl = pp[TT + a], Hl = pp[2 * TT + a];
              acc[a][0].fma(Pl, dv);
              acc[a][1].fma(Hl, vo);
              acc[a][2].fma(Pl, vo);
              acc[a][3].fma(Hl, dv);
              acc[a][4].fma(P, vo);
              acc[a][5].fma(P, dv);
              acc[a][6].fma(P, tt);
              acc[a][7].fma(P, qq);
            }
          }
        }
        // P of even rows and H of odd rows are symmetric about the equator, the
        // others antisymmetric: the even lane takes the north, the odd the south
#pragma unroll
        for (int a = 0; a < JG; ++a) {
          C2<R> c[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const C2<R> mine = acc[a][q].get(), other = shfl_xor_c(mine, 16);
            // (times +-1: exact)
            const C2<R> x = q == 1 || q == 3 ? other : mine, y = q == 1 || q == 3 ? mine : other;
            c[q] = cmk<R>(fma(x.x, sg, y.x), fma(x.y, sg, y.y));
          }
          const int jh = jg * JG + a;
          if (!live || jh >= JH) continue;
          const int j = par ? J - 1 - jh : jh;
          C2<R>* o = sfe + (((size_t)m * J + j) * K + k0 + kk) * SF_N;
          store_pair(o + SF_U, im_mul(c[0], rm) - c[1], im_mul(c[2], rm) + c[3]);
          store_pair(o + SF_VOR, c[4], c[5]);
          store_pair(o + SF_T, c[6], c[7]);
        }
      }
    }
  }
}

}  // namespace lbm
