// Spectral transforms on the reference array layouts: the building blocks of
// Spectral.grid_to_wave / wave_to_grid / hgrad / uv_to_vordiv / psichi_to_uv
// (spectral.py:159-276).  The fused ensemble stepper has its own kernels;
// these serve the drop-in Python API, setup and diagnostics.
#include "lbm_common.cuh"
#include "lbm_fft.cuh"

namespace lbm {

constexpr int FT_THREADS = 256;   // threads per block of the Fourier kernels
constexpr int FT_COLS = 32;       // columns (levels) per block

// grid[b][j][i][c] -> four[b][m][j][c] = jscale[j]/I rfft.  Block = (j, b,
// column chunk); the chunk's I x CC slab is staged transposed in shared
// memory, teams of R1 threads transform one column each.
template <typename R, int I>
__global__ void __launch_bounds__(FT_THREADS)
k_fourier_fwd(int J, int C, int M, const R* __restrict__ grid, const R* __restrict__ jscale,
              const C2<R>* __restrict__ twg, C2<R>* __restrict__ four) {
  constexpr int R1 = FftShape<I>::R1;
  constexpr int NTEAM = FT_THREADS / R1;
  constexpr int SCR = fft_team_scratch<I>();
  extern __shared__ unsigned char smraw[];
  C2<R>* tw = reinterpret_cast<C2<R>*>(smraw);
  C2<R>* scr = tw + I;                       // [NTEAM][SCR]
  C2<R>* outst = scr + NTEAM * SCR;          // [M][FT_COLS]
  R* slab = reinterpret_cast<R*>(outst + M * FT_COLS);  // [FT_COLS][I+1]
  const int j = blockIdx.x, b = blockIdx.y, c0 = blockIdx.z * FT_COLS;
  const int cc = min(FT_COLS, C - c0);
  const int tid = threadIdx.x;
  for (int p = tid; p < I; p += FT_THREADS) tw[p] = twg[p];
  const R* src = grid + ((size_t)b * J + j) * I * C;
  for (int idx = tid; idx < I * cc; idx += FT_THREADS) {
    const int i = idx / cc, c = idx % cc;
    slab[c * (I + 1) + i] = src[(size_t)i * C + c0 + c];
  }
  __syncthreads();
  const R scale = (jscale ? jscale[j] : R(1)) / R(I);
  const int team = tid / R1, t = tid % R1;
  for (int c = team; c < cc; c += NTEAM) {
    team_rfft_fwd<I>(t, slab + c * (I + 1), 1, scr + team * SCR, tw, M, scale,
                     [&](int m, C2<R> X) { outst[m * FT_COLS + c] = X; });
  }
  __syncthreads();
  for (int idx = tid; idx < M * cc; idx += FT_THREADS) {
    const int m = idx / cc, c = idx % cc;
    four[(((size_t)b * M + m) * J + j) * C + c0 + c] = outst[m * FT_COLS + c];
  }
}

template <typename R, int I>
__global__ void __launch_bounds__(FT_THREADS)
k_fourier_inv(int J, int C, int M, const C2<R>* __restrict__ four, const R* __restrict__ jscale,
              const C2<R>* __restrict__ twg, R* __restrict__ grid) {
  constexpr int R1 = FftShape<I>::R1;
  constexpr int NTEAM = FT_THREADS / R1;
  constexpr int SCR = fft_team_scratch<I>();
  extern __shared__ unsigned char smraw[];
  C2<R>* tw = reinterpret_cast<C2<R>*>(smraw);
  C2<R>* scr = tw + I;
  C2<R>* inst = scr + NTEAM * SCR;           // [FT_COLS][M]
  R* slab = reinterpret_cast<R*>(inst + M * FT_COLS);  // [FT_COLS][I+1]
  const int j = blockIdx.x, b = blockIdx.y, c0 = blockIdx.z * FT_COLS;
  const int cc = min(FT_COLS, C - c0);
  const int tid = threadIdx.x;
  for (int p = tid; p < I; p += FT_THREADS) tw[p] = twg[p];
  for (int idx = tid; idx < M * cc; idx += FT_THREADS) {
    const int m = idx / cc, c = idx % cc;
    inst[c * M + m] = four[(((size_t)b * M + m) * J + j) * C + c0 + c];
  }
  __syncthreads();
  const R scale = jscale ? jscale[j] : R(1);
  const int team = tid / R1, t = tid % R1;
  for (int c = team; c < cc; c += NTEAM) {
    const C2<R>* X = inst + c * M;
    team_rfft_inv<I>(t, [&](int m) { return X[m]; }, M, scr + team * SCR, tw,
                     slab + c * (I + 1), 1, scale);
  }
  __syncthreads();
  R* dst = grid + ((size_t)b * J + j) * I * C;
  for (int idx = tid; idx < I * cc; idx += FT_THREADS) {
    const int i = idx / cc, c = idx % cc;
    dst[(size_t)i * C + c0 + c] = slab[c * (I + 1) + i];
  }
}

// Legendre sums of the transform API.  One thread per output value (n or j, column):
// a block takes LG_NT consecutive values of one (m, batch, column chunk), walks the
// summation index in tiles of LG_T and stages the tile's table rows and column
// values in shared memory.  The order of each sum is the index's.
//
// FP64 is bound by its multiply-adds (about two per clock and SM): all lanes have
// to hold values, and one batch item has to spread over the SMs.  So the columns
// are cut evenly (20 stay one chunk, where fixed chunks of 16 left 38 % of the
// lanes idle) and the values of a chunk are dealt out flat, four warps a block.
// us at T42, 20 levels, before -> after: 32 members, analysis of two tables 559 -> 295,
// of one 292 -> 154, synthesis (mean of three calls) 411 -> 260; one member, analysis
// 56 -> 26, synthesis 65 -> 24.
constexpr int LG_NT = 128;      // threads of a block ...
constexpr int LG_NTMAX = 512;   // ... of the synthesis of many batch items
constexpr int LG_T = 32;        // summation indices per staged tile
constexpr int LG_CMAX = 32;     // columns of a chunk at most

inline int leg_cols(int C) {
  const int n = (C + LG_CMAX - 1) / LG_CMAX;
  return (C + n - 1) / n;
}
// Rows (n or j, of nrow) that nt consecutive values of cc columns touch at most.
LBM_HD int leg_rows(int cc, int nrow, int nt) {
  const int r = (nt + cc - 2) / cc + 1;
  return r < nrow ? r : nrow;
}

template <typename R> size_t leg_smem1(int cc, int nrow, int nt) {
  return 2 * (sizeof(C2<R>) * LG_T * (size_t)cc + sizeof(R) * leg_rows(cc, nrow, nt) * (LG_T + 1));
}
// Largest over the full chunks and the last one.
template <typename R> size_t leg_smem(int C, int CC, int nrow, int nt) {
  const size_t a = leg_smem1<R>(CC, nrow, nt),
               b = leg_smem1<R>(C - (C - 1) / CC * CC, nrow, nt);
  return a > b ? a : b;
}

// spec[b][m][n][c] (+)= nfac[n] (ca sum_j ta f_a + sb cb sum_j tb f_b)
template <typename R>
__global__ void __launch_bounds__(LG_NT)
k_leg_anal(int M, int J, int C, int CC, int nch, int z0, const C2<R>* __restrict__ fa,
           const R* __restrict__ ta, int ima, const C2<R>* __restrict__ fb,
           const R* __restrict__ tb, int imb, R sb, const R* __restrict__ nfac, int accumulate,
           C2<R>* __restrict__ spec) {
  extern __shared__ __align__(16) unsigned char smraw[];
  constexpr int TS = LG_T + 1;
  C2<R>* xs = reinterpret_cast<C2<R>*>(smraw);           // [2][LG_T][cc]
  const int m = blockIdx.x, b = blockIdx.y;
  const int z = z0 + (int)blockIdx.z, ch = z % nch, part = z / nch;
  const int c0 = ch * CC, cc = min(CC, C - c0), RR = leg_rows(cc, M, LG_NT);
  R* ts = reinterpret_cast<R*>(xs + 2 * LG_T * cc);      // [2][RR][TS]
  const int tid = threadIdx.x, v0 = part * LG_NT, v = v0 + tid;
  C2<R>* out = spec + ((size_t)b * M + m) * M * C + c0;
  if (!accumulate && v < m * cc) {                       // n < m: zeros
    const int n = v / cc;
    out[(size_t)n * C + v - n * cc] = cmk<R>(0, 0);
  }
  const int nval = (M - m) * cc;
  if (v0 >= nval) return;
  const bool act = v < nval;
  const int row = act ? v / cc : 0, c = act ? v - row * cc : 0, n = m + row;
  const int r0 = v0 / cc, nr = min(RR, M - m - r0);
  const C2<R>* ga = fa + ((size_t)b * M + m) * J * C + c0;
  const C2<R>* gb = fb ? fb + ((size_t)b * M + m) * J * C + c0 : nullptr;
  const size_t trow = ((size_t)m * M + m + r0) * J;
  C2<R> acc = cmk<R>(0, 0), accb = cmk<R>(0, 0);
  for (int j0 = 0; j0 < J; j0 += LG_T) {
    const int nj = min(LG_T, J - j0);
    __syncthreads();
    for (int x = tid; x < nj * cc; x += LG_NT) {
      const int jj = x / cc, q = x - jj * cc;
      const size_t g = (size_t)(j0 + jj) * C + q;
      xs[jj * cc + q] = ga[g];
      if (gb) xs[(LG_T + jj) * cc + q] = gb[g];
    }
    for (int x = tid; x < nr * LG_T; x += LG_NT) {
      const int r = x / LG_T, jj = x % LG_T;
      if (jj < nj) {
        ts[r * TS + jj] = ta[trow + (size_t)r * J + j0 + jj];
        if (gb) ts[(RR + r) * TS + jj] = tb[trow + (size_t)r * J + j0 + jj];
      }
    }
    __syncthreads();
    const C2<R>* x = xs + c;
    const R* t = ts + (row - r0) * TS;
    if (!act) continue;
    if (gb) {
#pragma unroll 4
      for (int jj = 0; jj < nj; ++jj) {
        cfma(acc, t[jj], x[jj * cc]);
        cfma(accb, t[RR * TS + jj], x[(LG_T + jj) * cc]);
      }
    } else {
#pragma unroll 4
      for (int jj = 0; jj < nj; ++jj) cfma(acc, t[jj], x[jj * cc]);
    }
  }
  if (!act) return;
  const R mm = R(m);
  if (ima) acc = im_mul(acc, mm);
  if (fb) {
    if (imb) accb = im_mul(accb, mm);
    acc = acc + accb * sb;
  }
  if (nfac) acc = acc * nfac[n];
  C2<R>* o = out + (size_t)n * C + c;
  if (accumulate) acc = acc + *o;
  *o = acc;
}

// (the factors of the staged coefficients are FP64 products too: large batches take
// LG_NTMAX values a block to stage less often: 32 members 400 -> 313 us)
// four[b][m][j][c] = sum_n ta[m][n][j] ca na[n] sa + sb sum_n tb cb nb[n] sb_
template <typename R>
__global__ void __launch_bounds__(LG_NTMAX)
k_leg_synth(int M, int J, int C, int CC, int nch, int z0, const C2<R>* __restrict__ sa,
            const R* __restrict__ ta, int ima, const R* __restrict__ na,
            const C2<R>* __restrict__ sbp, const R* __restrict__ tb, int imb,
            const R* __restrict__ nb, R sb, C2<R>* __restrict__ four) {
  extern __shared__ __align__(16) unsigned char smraw[];
  C2<R>* xs = reinterpret_cast<C2<R>*>(smraw);           // [2][LG_T][cc]
  const int m = blockIdx.x, b = blockIdx.y;
  const int z = z0 + (int)blockIdx.z, ch = z % nch, part = z / nch;
  const int c0 = ch * CC, cc = min(CC, C - c0), NT = blockDim.x,
            RR = leg_rows(cc, J, NT);
  R* ts = reinterpret_cast<R*>(xs + 2 * LG_T * cc);      // [2][LG_T][RR]
  const int tid = threadIdx.x, v0 = part * NT, v = v0 + tid, nval = J * cc;
  if (v0 >= nval) return;
  const bool act = v < nval;
  const int jj = act ? v / cc : 0, c = act ? v - jj * cc : 0;
  const int r0 = v0 / cc, nr = min(RR, J - r0);
  const R mm = R(m);
  C2<R> acc = cmk<R>(0, 0);
  for (int n0 = m; n0 < M; n0 += LG_T) {
    const int nn = min(LG_T, M - n0);
    __syncthreads();
    for (int x = tid; x < nn * cc; x += NT) {
      const int y = x / cc, q = x - y * cc, n = n0 + y;
      const size_t g = (((size_t)b * M + m) * M + n) * C + c0 + q;
      C2<R> va = sa[g];
      if (ima) va = im_mul(va, mm);
      if (na) va = va * na[n];
      xs[y * cc + q] = va;
      if (sbp) {
        C2<R> vb = sbp[g];
        if (imb) vb = im_mul(vb, mm);
        if (nb) vb = vb * nb[n];
        xs[(LG_T + y) * cc + q] = vb * sb;
      }
    }
    for (int x = tid; x < nn * nr; x += NT) {
      const int y = x / nr, r = x - y * nr;
      const size_t g = ((size_t)m * M + n0 + y) * J + r0 + r;
      ts[y * RR + r] = ta[g];
      if (sbp) ts[(LG_T + y) * RR + r] = tb[g];
    }
    __syncthreads();
    const C2<R>* x = xs + c;
    const R* t = ts + (jj - r0);
    if (!act) continue;
    if (sbp) {
#pragma unroll 4
      for (int y = 0; y < nn; ++y) {
        cfma(acc, t[y * RR], x[y * cc]);
        cfma(acc, t[(LG_T + y) * RR], x[(LG_T + y) * cc]);
      }
    } else {
#pragma unroll 4
      for (int y = 0; y < nn; ++y) cfma(acc, t[y * RR], x[y * cc]);
    }
  }
  if (act) four[(((size_t)b * M + m) * J + jj) * C + c0 + c] = acc;
}

// The same sums with the column values of a whole sum staged once: a block takes all
// values of one (m, batch, LG_COLS columns), a thread every LG_ROWS-th n or j of one
// column, its table rows read in place.  Fewer stagings and half the shared-memory
// reads per product, but lanes without a column idle, a block walks its rows in
// turn, and shared memory holds 454 indices in FP64.  leg_whole() gives the sizes
// at which this form is the faster one; the results are the same bits.
constexpr int LG_COLS = 16;     // columns of a block
constexpr int LG_ROWS = 16;     // thread rows (n or j)

// spec[b][m][n][c] (+)= nfac[n] (ca sum_j ta f_a + sb cb sum_j tb f_b)
template <typename R>
__global__ void __launch_bounds__(LG_COLS * LG_ROWS)
k_leg_anal16(int M, int J, int C, const C2<R>* __restrict__ fa, const R* __restrict__ ta,
           int ima, const C2<R>* __restrict__ fb, const R* __restrict__ tb, int imb, R sb,
           const R* __restrict__ nfac, int accumulate, C2<R>* __restrict__ spec) {
  extern __shared__ unsigned char smraw[];
  C2<R>* sa = reinterpret_cast<C2<R>*>(smraw);   // [J][LG_COLS]
  C2<R>* sbb = sa + J * LG_COLS;
  const int m = blockIdx.x, b = blockIdx.y, c0 = blockIdx.z * LG_COLS;
  const int cc = min(LG_COLS, C - c0);
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * LG_COLS + tx;
  for (int idx = tid; idx < J * LG_COLS; idx += LG_COLS * LG_ROWS) {
    const int jj = idx / LG_COLS, c = idx % LG_COLS;
    const size_t g = (((size_t)b * M + m) * J + jj) * C + c0 + c;
    sa[idx] = (c < cc) ? fa[g] : cmk<R>(0, 0);
    if (fb) sbb[idx] = (c < cc) ? fb[g] : cmk<R>(0, 0);
  }
  __syncthreads();
  if (tx >= cc) return;
  const R mm = R(m);
  for (int n = ty; n < M; n += LG_ROWS) {
    const size_t o = (((size_t)b * M + m) * M + n) * C + c0 + tx;
    if (n < m) {
      if (!accumulate) spec[o] = cmk<R>(0, 0);
      continue;
    }
    const R* pa = ta + ((size_t)m * M + n) * J;
    C2<R> acc = cmk<R>(0, 0), accb = cmk<R>(0, 0);
    for (int jj = 0; jj < J; ++jj) cfma(acc, pa[jj], sa[jj * LG_COLS + tx]);
    if (ima) acc = im_mul(acc, mm);
    if (fb) {
      const R* pb = tb + ((size_t)m * M + n) * J;
      for (int jj = 0; jj < J; ++jj) cfma(accb, pb[jj], sbb[jj * LG_COLS + tx]);
      if (imb) accb = im_mul(accb, mm);
      acc = acc + accb * sb;
    }
    if (nfac) acc = acc * nfac[n];
    if (accumulate) acc = acc + spec[o];
    spec[o] = acc;
  }
}

// four[b][m][j][c] = sum_n ta[m][n][j] ca na[n] sa + sb sum_n tb cb nb[n] sb_
template <typename R>
__global__ void __launch_bounds__(LG_COLS * LG_ROWS)
k_leg_synth16(int M, int J, int C, const C2<R>* __restrict__ sa, const R* __restrict__ ta,
            int ima, const R* __restrict__ na, const C2<R>* __restrict__ sbp,
            const R* __restrict__ tb, int imb, const R* __restrict__ nb, R sb,
            C2<R>* __restrict__ four) {
  extern __shared__ unsigned char smraw[];
  C2<R>* xa = reinterpret_cast<C2<R>*>(smraw);   // [M][LG_COLS]
  C2<R>* xb = xa + M * LG_COLS;
  const int m = blockIdx.x, b = blockIdx.y, c0 = blockIdx.z * LG_COLS;
  const int cc = min(LG_COLS, C - c0);
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * LG_COLS + tx;
  const R mm = R(m);
  for (int idx = tid; idx < M * LG_COLS; idx += LG_COLS * LG_ROWS) {
    const int n = idx / LG_COLS, c = idx % LG_COLS;
    C2<R> va = cmk<R>(0, 0), vb = cmk<R>(0, 0);
    if (c < cc && n >= m) {
      const size_t g = (((size_t)b * M + m) * M + n) * C + c0 + c;
      va = sa[g];
      if (ima) va = im_mul(va, mm);
      if (na) va = va * na[n];
      if (sbp) {
        vb = sbp[g];
        if (imb) vb = im_mul(vb, mm);
        if (nb) vb = vb * nb[n];
        vb = vb * sb;
      }
    }
    xa[idx] = va;
    xb[idx] = vb;
  }
  __syncthreads();
  if (tx >= cc) return;
  for (int jj = ty; jj < J; jj += LG_ROWS) {
    C2<R> acc = cmk<R>(0, 0);
    for (int n = m; n < M; ++n) {
      cfma(acc, ta[((size_t)m * M + n) * J + jj], xa[n * LG_COLS + tx]);
      if (sbp) cfma(acc, tb[((size_t)m * M + n) * J + jj], xb[n * LG_COLS + tx]);
    }
    four[(((size_t)b * M + m) * J + jj) * C + c0 + tx] = acc;
  }
}

template <typename R, int I>
int launch_fourier(bool fwd, int B, int J, int C, int M, const void* in, const void* js,
                   const void* tw, void* out, cudaStream_t st) {
  constexpr int R1 = FftShape<I>::R1;
  constexpr int NTEAM = FT_THREADS / R1;
  const size_t smem = sizeof(C2<R>) * (I + NTEAM * fft_team_scratch<I>() + M * FT_COLS) +
                      sizeof(R) * FT_COLS * (I + 1);
  dim3 grid(J, B, (C + FT_COLS - 1) / FT_COLS);
  if (fwd) {
    allow_smem(k_fourier_fwd<R, I>);
    k_fourier_fwd<R, I><<<grid, FT_THREADS, smem, st>>>(
        J, C, M, (const R*)in, (const R*)js, (const C2<R>*)tw, (C2<R>*)out);
  } else {
    allow_smem(k_fourier_inv<R, I>);
    k_fourier_inv<R, I><<<grid, FT_THREADS, smem, st>>>(
        J, C, M, (const C2<R>*)in, (const R*)js, (const C2<R>*)tw, (R*)out);
  }
  LBM_LAUNCH_CHECK();
  return LBM_OK;
}

template <typename R>
int fourier_dispatch(bool fwd, int B, int J, int I, int C, int nmax, const void* in,
                     const void* js, const void* tw, void* out, cudaStream_t st) {
  const int M = nmax + 1;
  if (B < 1 || J < 2 || C < 1 || M < 1 || 2 * M > I || !in || !tw || !out) return LBM_ERR_ARG;
  switch (I) {
    case 64: return launch_fourier<R, 64>(fwd, B, J, C, M, in, js, tw, out, st);
    case 128: return launch_fourier<R, 128>(fwd, B, J, C, M, in, js, tw, out, st);
    case 256: return launch_fourier<R, 256>(fwd, B, J, C, M, in, js, tw, out, st);
    default: return LBM_ERR_ARG;
  }
}

// Launches of nz chunks and value parts, at most LG_ZMAX in the third dimension of a
// grid: one launch up to 95 thousand columns at T85.
constexpr int LG_ZMAX = 65535;
template <typename F> void leg_launches(int M, int B, long nz, F launch) {
  for (long z = 0; z < nz; z += LG_ZMAX)
    launch(dim3(M, B, (unsigned)(nz - z < LG_ZMAX ? nz - z : LG_ZMAX)), (int)z);
}

// Whether the 16-column form takes a sum: batches that fill the SMs, and columns that
// fill its chunks (at most `fill` lanes per 100 columns; idle lanes cost as much as
// others).  us, flat values -> 16-column form.  FP32: T42, 32 items of 64 columns,
// analysis of one table 97 -> 66, of two 140 -> 123, synthesis 95 -> 64 and 130 -> 113;
// T21, 128 items of 48, 51 -> 30 and 64 -> 36.  FP64: T42, 32 items of 64 columns,
// synthesis 476 -> 446 and 989 -> 897.  The flat form keeps, FP32: T21, 128 items of 20
// columns, 23 (21) and T42, four items of 16, 6 (9); FP64: fewer items, more idle
// lanes, and every analysis (T42, 32 items of 64: 448 (509)).
template <typename R> bool leg_whole(bool synth, bool two, int n, int B, int C) {
  const int nch = (C + LG_COLS - 1) / LG_COLS;
  if (nch > 65535 || sizeof(C2<R>) * 2 * (size_t)n * LG_COLS > SMEM_BLOCK) return false;
  if (sizeof(R) == 8) return synth && 100 * LG_COLS * nch <= 115 * C && (long)B * nch >= 40;
  const int fill = synth ? (two ? 150 : 190) : (two ? 130 : 150);
  const long most = synth ? (two ? 40 : 16) : 10;
  return 100 * (long)LG_COLS * nch <= (long)fill * C && (long)B * nch >= most;
}

template <typename R>
static int leg_anal(int B, int nmax, int J, int C, const void* fa, const void* ta, int ima,
                    const void* fb, const void* tb, int imb, double sb, const void* nfac,
                    int acc, void* spec, cudaStream_t st) {
  const int M = nmax + 1;
  if (B < 1 || M < 1 || J < 2 || C < 1 || !fa || !ta || !spec || (fb && !tb))
    return LBM_ERR_ARG;
  if (leg_whole<R>(false, fb != nullptr, J, B, C)) {
    allow_smem(k_leg_anal16<R>);
    k_leg_anal16<R><<<dim3(M, B, (C + LG_COLS - 1) / LG_COLS), dim3(LG_COLS, LG_ROWS),
                      sizeof(C2<R>) * 2 * J * LG_COLS, st>>>(
        M, J, C, (const C2<R>*)fa, (const R*)ta, ima, (const C2<R>*)fb, (const R*)tb, imb, R(sb),
        (const R*)nfac, acc, (C2<R>*)spec);
    LBM_LAUNCH_CHECK();
    return LBM_OK;
  }
  const int CC = leg_cols(C), nch = (C + CC - 1) / CC;
  const long nz = (long)nch * ((M * CC + LG_NT - 1) / LG_NT);
  const size_t smem = leg_smem<R>(C, CC, M, LG_NT);
  allow_smem(k_leg_anal<R>);
  leg_launches(M, B, nz, [&](dim3 grid, int z0) {
    k_leg_anal<R><<<grid, LG_NT, smem, st>>>(
        M, J, C, CC, nch, z0, (const C2<R>*)fa, (const R*)ta, ima, (const C2<R>*)fb,
        (const R*)tb, imb, R(sb), (const R*)nfac, acc, (C2<R>*)spec);
  });
  LBM_LAUNCH_CHECK();
  return LBM_OK;
}

template <typename R>
static int leg_synth(int B, int nmax, int J, int C, const void* sa, const void* ta, int ima,
                     const void* na, const void* sbp, const void* tb, int imb, const void* nb,
                     double sb, void* four, cudaStream_t st) {
  const int M = nmax + 1;
  if (B < 1 || M < 1 || J < 2 || C < 1 || !sa || !ta || !four || (sbp && !tb))
    return LBM_ERR_ARG;
  if (leg_whole<R>(true, sbp != nullptr, M, B, C)) {
    allow_smem(k_leg_synth16<R>);
    k_leg_synth16<R><<<dim3(M, B, (C + LG_COLS - 1) / LG_COLS), dim3(LG_COLS, LG_ROWS),
                       sizeof(C2<R>) * 2 * M * LG_COLS, st>>>(
        M, J, C, (const C2<R>*)sa, (const R*)ta, ima, (const R*)na, (const C2<R>*)sbp,
        (const R*)tb, imb, (const R*)nb, R(sb), (C2<R>*)four);
    LBM_LAUNCH_CHECK();
    return LBM_OK;
  }
  const int CC = leg_cols(C), nch = (C + CC - 1) / CC;
  const int big = (J * CC + LG_NTMAX - 1) / LG_NTMAX;
  // LG_NTMAX values a block where those blocks are eight per SM; three for two tables
  // in FP64, whose staged factors cost most (us with 128 -> 512, T42, two tables: one
  // item of 100 columns 83 -> 64, four of 31 105 -> 90), but not for a few columns.
  // (One column of many latitudes in FP64: that many table rows exceed a block.)
  const int per_sm = sizeof(R) == 8 && sbp && CC >= 8 ? 3 : 8;
  const int nt = (long)M * B * nch * big >= per_sm * FILL_SMS &&
                         leg_smem<R>(C, CC, J, LG_NTMAX) <= SMEM_BLOCK
                     ? LG_NTMAX
                     : LG_NT;
  const long nz = (long)nch * ((J * CC + nt - 1) / nt);
  const size_t smem = leg_smem<R>(C, CC, J, nt);
  allow_smem(k_leg_synth<R>);
  leg_launches(M, B, nz, [&](dim3 grid, int z0) {
    k_leg_synth<R><<<grid, nt, smem, st>>>(
        M, J, C, CC, nch, z0, (const C2<R>*)sa, (const R*)ta, ima, (const R*)na,
        (const C2<R>*)sbp, (const R*)tb, imb, (const R*)nb, R(sb), (C2<R>*)four);
  });
  LBM_LAUNCH_CHECK();
  return LBM_OK;
}

}  // namespace lbm

using namespace lbm;

extern "C" {

int lbm_fourier_forward(int prec, int batch, int nlat, int nlon, int ncol, int nmax,
                        const void* grid, const void* jscale, const void* tw, void* four,
                        void* stream) {
  if (prec == LBM_F64)
    return fourier_dispatch<double>(true, batch, nlat, nlon, ncol, nmax, grid, jscale, tw,
                                    four, (cudaStream_t)stream);
  if (prec == LBM_F32)
    return fourier_dispatch<float>(true, batch, nlat, nlon, ncol, nmax, grid, jscale, tw, four,
                                   (cudaStream_t)stream);
  return LBM_ERR_ARG;
}

int lbm_fourier_inverse(int prec, int batch, int nlat, int nlon, int ncol, int nmax,
                        const void* four, const void* jscale, const void* tw, void* grid,
                        void* stream) {
  if (prec == LBM_F64)
    return fourier_dispatch<double>(false, batch, nlat, nlon, ncol, nmax, four, jscale, tw,
                                    grid, (cudaStream_t)stream);
  if (prec == LBM_F32)
    return fourier_dispatch<float>(false, batch, nlat, nlon, ncol, nmax, four, jscale, tw,
                                   grid, (cudaStream_t)stream);
  return LBM_ERR_ARG;
}

int lbm_legendre_analysis(int prec, int batch, int nmax, int nlat, int ncol, const void* fa,
                          const void* ta, int ima, const void* fb, const void* tb, int imb,
                          double sb, const void* nfac, int accumulate, void* spec,
                          void* stream) {
  if (prec == LBM_F64)
    return leg_anal<double>(batch, nmax, nlat, ncol, fa, ta, ima, fb, tb, imb, sb, nfac,
                            accumulate, spec, (cudaStream_t)stream);
  if (prec == LBM_F32)
    return leg_anal<float>(batch, nmax, nlat, ncol, fa, ta, ima, fb, tb, imb, sb, nfac,
                           accumulate, spec, (cudaStream_t)stream);
  return LBM_ERR_ARG;
}

int lbm_legendre_synthesis(int prec, int batch, int nmax, int nlat, int ncol, const void* sa,
                           const void* ta, int ima, const void* na, const void* sb_,
                           const void* tb, int imb, const void* nb, double sb, void* four,
                           void* stream) {
  if (prec == LBM_F64)
    return leg_synth<double>(batch, nmax, nlat, ncol, sa, ta, ima, na, sb_, tb, imb, nb, sb,
                             four, (cudaStream_t)stream);
  if (prec == LBM_F32)
    return leg_synth<float>(batch, nmax, nlat, ncol, sa, ta, ima, na, sb_, tb, imb, nb, sb,
                            four, (cudaStream_t)stream);
  return LBM_ERR_ARG;
}

}  // extern "C"
