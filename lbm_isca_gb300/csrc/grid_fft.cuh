// FP64 longitude transforms of the split grid-point step (included by
// stepper.cu): k_ifft (sf, sfs -> grid6) and k_ffft (grid9 -> af, afs) around
// the column algebra k_alg, on the row layouts of grid_split.cuh.
//
// GB300 retires two FP64 FMAs per SM clock, so these kernels are bound by the
// FP64 pipe and by how many SMs have work.  A real FFT (lbm_fft.cuh: one team
// of R1 threads per row, about 1,500 FP64 instructions a row at 128 points)
// takes fewer FP64 operations than the folded dense DFT of the FP32 kernels
// (2,750), and one row per team lets a block cover a few levels only: one
// member fills the chip (T42L20: 384 blocks against the 64 of the fused
// k_grid), and 40-70 KB of shared memory keep two to four blocks per SM
// resident where k_grid's level ring takes 185 KB.
// Measured per step at T42L20 (grid part: these two and k_alg): 1 member
// 675 -> 145 us (k_ifft 38, k_alg 47, k_ffft 60), 32 members 9.27 -> 2.95 ms
// (0.80, 0.89, 1.26).
#pragma once

namespace lbm {

// Levels per block of the two kernels: one team per row.
template <int I> struct GridFft {
  static constexpr int R1 = FftShape<I>::R1;
  static constexpr int SCR = fft_team_scratch<I>();
  static constexpr int LI = I == 256 ? 2 : 4;      // levels per k_ifft block (6 rows each)
  static constexpr int LF = I == 256 ? 2 : 4;      // levels per k_ffft block (9 rows each)
  static constexpr int TI = 6 * LI, TF = 9 * LF;   // teams
  static constexpr int NTI = ((TI * R1 + 31) / 32) * 32;
  static constexpr int NTF = ((TF * R1 + 31) / 32) * 32;
  static __host__ __device__ int row_stride(int M) { return M | 1; }   // odd: no bank conflicts
  template <typename R> static size_t ifft_smem(int M) {
    return sizeof(C2<R>) * (size_t)(I + TI * SCR + TI * row_stride(M));
  }
  template <typename R> static size_t ffft_smem(int M) {
    return sizeof(C2<R>) * (size_t)(I + TF * SCR + TF * row_stride(M));
  }
};

// Longitude synthesis: block (latitude, chunk, member), chunk 0 the six
// surface rows (pi, pi_x, pi_y, U-, V-, D-sum), chunk c > 0 levels
// (c - 1) LI .. of the six fields.
template <typename R, int I>
__global__ void __launch_bounds__(GridFft<I>::NTI) k_ifft(SD<R> d) {
  using G = GridFft<I>;
  const int j = blockIdx.x, e = blockIdx.z;
  const int J = d.J, K = d.K, M = d.M, RS = G::row_stride(M);
  const int tid = threadIdx.x, team = tid / G::R1, t = tid % G::R1;
  extern __shared__ unsigned char smraw[];
  C2<R>* tw = reinterpret_cast<C2<R>*>(smraw);
  C2<R>* scr = tw + I;
  C2<R>* X = scr + G::TI * G::SCR;                       // [rows][RS]
  for (int p = tid; p < I; p += G::NTI) tw[p] = d.tw[p];
  const R rcos = d.jfac[JF_RCOS * J + j];
  const bool surf = blockIdx.y == 0;
  const int k0 = surf ? 0 : ((int)blockIdx.y - 1) * G::LI;
  const int nr = surf ? 6 : SF_N * min(G::LI, K - k0);
  if (surf) {
    for (int x = tid; x < M * SFS_N; x += G::NTI) {
      const int m = x / SFS_N, f = x - m * SFS_N;
      const C2<R> v = d.sfs[(((size_t)e * M + m) * J + j) * SFS_N + f];
      if (f == SFS_PI) {
        X[m] = v;
        X[RS + m] = im_mul(v, R(m));
      } else {
        X[(f + 1) * RS + m] = v;
      }
    }
  } else {
    const C2<R>* src = d.sf + (((size_t)e * M * J + j) * K + k0) * SF_N;
    const size_t ms = (size_t)J * K * SF_N;
    const FastDiv fr(nr);
    for (int x = tid; x < M * nr; x += G::NTI) {
      const int m = fr.div(x), r = x - m * nr;
      X[r * RS + m] = src[m * ms + r];
    }
  }
  __syncthreads();
  if (team >= nr) return;                                // whole teams; none waits below
  R* row = d.grid6 + (((size_t)e * J + j) * (6 + 6 * K) + (surf ? 0 : 6 + SF_N * k0) + team) * I;
  // rows in 1 / (a cos): pi_x, pi_y, U-, V-sum; u, v of a level
  const int f = team % SF_N;
  const bool scaled = surf ? (team >= 1 && team <= 4) : (f == SF_U || f == SF_V);
  const C2<R>* x = X + team * RS;
  team_rfft_inv<I>(t, [&](int m) { return x[m]; }, M, scr + team * G::SCR, tw, row, 1,
                   scaled ? rcos : R(1));
}

// Longitude analysis: block (latitude, chunk, member), chunk 0 the two
// surface rows, chunk c > 0 levels (c - 1) LF ..: one team per grid row, the
// rows of a level combined (wg X(gt) - wd i m X(xu), ...) on the way out.
template <typename R, int I>
__global__ void __launch_bounds__(GridFft<I>::NTF) k_ffft(SD<R> d) {
  using G = GridFft<I>;
  const int j = blockIdx.x, e = blockIdx.z;
  const int J = d.J, K = d.K, M = d.M, RS = G::row_stride(M);
  const int tid = threadIdx.x, team = tid / G::R1, t = tid % G::R1;
  extern __shared__ unsigned char smraw[];
  C2<R>* tw = reinterpret_cast<C2<R>*>(smraw);
  C2<R>* scr = tw + I;
  C2<R>* Y = scr + G::TF * G::SCR;                       // [rows][RS]
  for (int p = tid; p < I; p += G::NTF) tw[p] = d.tw[p];
  __syncthreads();
  const R wg = d.jfac[JF_GW * J + j] / R(I), wd = d.jfac[JF_GWDELC * J + j] / R(I);
  const bool surf = blockIdx.y == 0;
  const int k0 = surf ? 0 : ((int)blockIdx.y - 1) * G::LF;
  const int lc = min(G::LF, K - k0), nr = surf ? 2 : 9 * lc;
  if (team < nr) {
    const R* row = d.grid9 + (((size_t)e * J + j) * (2 + 9 * K) + (surf ? 0 : 2 + 9 * k0) + team) * I;
    // rows gt xu g yu fu fv ke xv yv; the surface rows take wg
    const int f = team % 9;
    const R w = (surf || f == 0 || f == 2 || f == 6) ? wg : wd;
    C2<R>* y = Y + team * RS;
    team_rfft_fwd<I>(t, row, 1, scr + team * G::SCR, tw, M, w, [&](int m, C2<R> v) { y[m] = v; });
  }
  __syncthreads();
  if (surf) {
    for (int x = tid; x < M * 2; x += G::NTF) {
      const int m = x >> 1, f = x & 1;
      d.afs[(((size_t)e * M + m) * J + j) * 2 + f] = Y[f * RS + m];
    }
    return;
  }
  C2<R>* out = d.af + (((size_t)e * M * J + j) * K + k0) * AF_N;
  const size_t ms = (size_t)J * K * AF_N;
  const int no = lc * AF_N;
  const FastDiv fo(no), fa(AF_N);
  for (int x = tid; x < M * no; x += G::NTF) {
    const int m = fo.div(x), r = x - m * no, l = fa.div(r), a = r - l * AF_N;
    const C2<R>* y = Y + (9 * l) * RS + m;
    C2<R> v;
    switch (a) {
      case AF_FU: v = y[4 * RS]; break;
      case AF_FV: v = y[5 * RS]; break;
      case AF_KE: v = y[6 * RS]; break;
      case AF_T: v = y[0] - im_mul(y[RS], R(m)); break;
      case AF_XV: v = y[7 * RS]; break;
      case AF_Q: v = y[2 * RS] - im_mul(y[3 * RS], R(m)); break;
      default: v = y[8 * RS]; break;
    }
    out[m * ms + r] = v;
  }
}

}  // namespace lbm
