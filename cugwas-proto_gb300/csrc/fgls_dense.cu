// FP64 dense kernels: tiled DGEMM for products too small for the digit form
// (fgls_digit_gemm.cu), blocked lower Cholesky (the reference's dpotrf of M, src/fgls_chol.c:252-271) and
// blocked lower-triangular solve X := L^-1 X (the reference's per-block
// dtrsm, src/fgls_chol.c:365-368 and cublasDtrsm in
// src/fgls_chol_gpu.c:543-555).
//
// GB300 executes FP64 at a small fraction of its FP32/tensor rate, so these
// kernels are FP64-issue-bound by design: tiles are sized to keep the FP64
// pipe fed from shared memory, not to chase memory bandwidth.
#include <algorithm>

#include "fgls_common.cuh"
#include "fgls_digit_gemm.cuh"
#include "fgls_kernels.cuh"

namespace fgls {

namespace {

constexpr int GM = 64, GN = 64, GK = 16;  // DGEMM CTA tile
constexpr int GT = 256;                   // threads: 16 x 16, 4 x 4 outputs each

// op(A)(i, k) for column-major A
__device__ __forceinline__ double ldA(const double* A, long long lda, bool tA, int i, int k) {
  return tA ? A[k + (long long)i * lda] : A[i + (long long)k * lda];
}

template <bool TA, bool TB, bool LOWER>
__global__ void __launch_bounds__(GT) dgemm_kernel(int M, int N, int K, double alpha,
                                                   const double* __restrict__ A, long long lda,
                                                   const double* __restrict__ B, long long ldb,
                                                   double beta, double* __restrict__ C,
                                                   long long ldc) {
  const int bi = blockIdx.x, bj = blockIdx.y;
  if (LOWER && bj > bi) return;  // tile strictly above the diagonal (square C, GM == GN)
  if (gridDim.z > 1) {
    // split K: slice z of the K range into its own M x N partial (ldc = M)
    const int kc = (K + (int)gridDim.z - 1) / (int)gridDim.z;
    const int k0 = (int)blockIdx.z * kc;
    K = max(0, min(K - k0, kc));
    A += TA ? (long long)k0 : (long long)k0 * lda;
    B += TB ? (long long)k0 * ldb : (long long)k0;
    C += (long long)blockIdx.z * ldc * N;
  }
  const int i0 = bi * GM, j0 = bj * GN;
  __shared__ double As[2][GK][GM + 1];
  __shared__ double Bs[2][GK][GN + 1];
  const int tid = threadIdx.x;
  const int tx = tid % 16, ty = tid / 16;
  double acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int b = 0; b < 4; b++) acc[a][b] = 0.0;

  // each thread loads 4 A and 4 B elements per k-tile
  double ra[4], rb[4];
  auto load_regs = [&](int k0) {
#pragma unroll
    for (int r = 0; r < 4; r++) {
      int e = tid + r * GT;  // 0..1023 over a GM x GK tile
      int ii, kk;
      if (!TA) { ii = e % GM; kk = e / GM; } else { kk = e % GK; ii = e / GK; }
      int gi = i0 + ii, gk = k0 + kk;
      ra[r] = (gi < M && gk < K) ? ldA(A, lda, TA, gi, gk) : 0.0;
      int jj, kb;
      if (!TB) { kb = e % GK; jj = e / GK; } else { jj = e % GN; kb = e / GN; }
      int gj = j0 + jj, gkb = k0 + kb;
      double v = 0.0;
      if (gj < N && gkb < K) v = TB ? B[gj + (long long)gkb * ldb] : B[gkb + (long long)gj * ldb];
      rb[r] = v;
    }
  };
  auto store_smem = [&](int buf) {
#pragma unroll
    for (int r = 0; r < 4; r++) {
      int e = tid + r * GT;
      int ii, kk;
      if (!TA) { ii = e % GM; kk = e / GM; } else { kk = e % GK; ii = e / GK; }
      As[buf][kk][ii] = ra[r];
      int jj, kb;
      if (!TB) { kb = e % GK; jj = e / GK; } else { jj = e % GN; kb = e / GN; }
      Bs[buf][kb][jj] = rb[r];
    }
  };

  const int nk = (K + GK - 1) / GK;
  if (nk > 0) {
    load_regs(0);
    store_smem(0);
  }
  __syncthreads();
  for (int kt = 0; kt < nk; kt++) {
    const int buf = kt & 1;
    if (kt + 1 < nk) load_regs((kt + 1) * GK);
#pragma unroll
    for (int k = 0; k < GK; k++) {
      double a[4], b[4];
#pragma unroll
      for (int r = 0; r < 4; r++) a[r] = As[buf][k][ty + 16 * r];
#pragma unroll
      for (int c = 0; c < 4; c++) b[c] = Bs[buf][k][tx + 16 * c];
#pragma unroll
      for (int r = 0; r < 4; r++)
#pragma unroll
        for (int c = 0; c < 4; c++) acc[r][c] = fma(a[r], b[c], acc[r][c]);
    }
    if (kt + 1 < nk) store_smem(buf ^ 1);
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < 4; r++) {
    int gi = i0 + ty + 16 * r;
    if (gi >= M) continue;
#pragma unroll
    for (int c = 0; c < 4; c++) {
      int gj = j0 + tx + 16 * c;
      if (gj >= N) continue;
      double* cp = C + gi + (long long)gj * ldc;
      double v = alpha * acc[r][c];
      if (beta != 0.0) v = fma(beta, *cp, v);
      *cp = v;
    }
  }
}

// The same product on 32 x 8 tiles, for outputs of less than a wave of 64 x 64
// tiles: an SM issues about two FP64 FMAs a clock, so a 64 x 64 tile takes 1.0 us
// per element of K on one SM while the others idle (301 x 74 x 301: 135 us; on
// 100 tiles of 32 x 8 20 us).
constexpr int SM_ = 32, SN_ = 8, SK_ = 32, ST_ = 128;
template <bool TA, bool TB>
__global__ void __launch_bounds__(ST_) dgemm_small_kernel(int M, int N, int K, double alpha, const double* __restrict__ A,
                                                          long long lda, const double* __restrict__ B, long long ldb,
                                                          double beta, double* __restrict__ C, long long ldc) {
  __shared__ double As[2][SK_][SM_ + 1], Bs[2][SK_][SN_ + 1];
  const int i0 = blockIdx.x * SM_, j0 = blockIdx.y * SN_;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  double ra[8], rb[2], acc[2] = {0.0, 0.0};
  auto load = [&](int k0) {
#pragma unroll
    for (int r = 0; r < 8; r++) {
      const int ii = TA ? ty + 4 * r : tx, kk = TA ? tx : ty + 4 * r;
      ra[r] = (i0 + ii < M && k0 + kk < K) ? ldA(A, lda, TA, i0 + ii, k0 + kk) : 0.0;
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const int e = threadIdx.x + r * ST_;
      const int jj = TB ? e % SN_ : e / SK_, kk = TB ? e / SN_ : e % SK_;
      rb[r] = (j0 + jj < N && k0 + kk < K) ? ldA(B, ldb, !TB, j0 + jj, k0 + kk) : 0.0;
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int r = 0; r < 8; r++) As[buf][TA ? tx : ty + 4 * r][TA ? ty + 4 * r : tx] = ra[r];
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const int e = threadIdx.x + r * ST_;
      Bs[buf][TB ? e / SN_ : e % SK_][TB ? e % SN_ : e / SK_] = rb[r];
    }
  };
  const int nk = (K + SK_ - 1) / SK_;
  if (nk > 0) {
    load(0);
    store(0);
  }
  __syncthreads();
  for (int kt = 0; kt < nk; kt++) {
    const int buf = kt & 1;
    if (kt + 1 < nk) load((kt + 1) * SK_);
#pragma unroll
    for (int k = 0; k < SK_; k++) {
      const double a = As[buf][k][tx];
      acc[0] = fma(a, Bs[buf][k][2 * ty], acc[0]);
      acc[1] = fma(a, Bs[buf][k][2 * ty + 1], acc[1]);
    }
    if (kt + 1 < nk) store(buf ^ 1);
    __syncthreads();
  }
#pragma unroll
  for (int u = 0; u < 2; u++) {
    const int i = i0 + tx, j = j0 + 2 * ty + u;
    if (i >= M || j >= N) continue;
    double* cp = C + i + (long long)j * ldc;
    const double v = alpha * acc[u];
    *cp = beta != 0.0 ? fma(beta, *cp, v) : v;
  }
}

template <bool LOWER>
cudaError_t launch_dgemm(cudaStream_t s, bool tA, bool tB, int M, int N, int K, double alpha,
                         const double* A, long long lda, const double* B, long long ldb,
                         double beta, double* C, long long ldc) {
  if (M <= 0 || N <= 0) return cudaSuccess;
  dim3 grid(ceil_div(M, GM), ceil_div(N, GN));
  if (!LOWER && grid.x * grid.y < 152) {
    const dim3 sg(ceil_div(M, SM_), ceil_div(N, SN_));
    if (!tA && !tB) dgemm_small_kernel<false, false><<<sg, ST_, 0, s>>>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
    else if (!tA) dgemm_small_kernel<false, true><<<sg, ST_, 0, s>>>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
    else if (!tB) dgemm_small_kernel<true, false><<<sg, ST_, 0, s>>>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
    else dgemm_small_kernel<true, true><<<sg, ST_, 0, s>>>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
    note_launch();
    return cudaGetLastError();
  }
  if (!tA && !tB) dgemm_kernel<false, false, LOWER><<<grid, GT, 0, s>>>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
  else if (!tA && tB) dgemm_kernel<false, true, LOWER><<<grid, GT, 0, s>>>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
  else if (tA && !tB) dgemm_kernel<true, false, LOWER><<<grid, GT, 0, s>>>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
  else dgemm_kernel<true, true, LOWER><<<grid, GT, 0, s>>>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
  note_launch();
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Diagonal-block kernels (NB = 128).
// ---------------------------------------------------------------------------
constexpr int NB = 128;       // block size of trsm
constexpr int SCB = 64;       // RHS columns per CTA in the diagonal solve
constexpr int DT = 256;       // threads of the diagonal kernels
constexpr int PB = 64;        // diagonal block of potrf and of the inverse
constexpr int PO = 512;       // outer panel of potrf, base block of the inverse

// Cholesky factor of a 64 x 64 block and its inverse, one CTA of eight warps
// (FACTOR = false: the inverse alone, Ls and rdiag given).
//   Ls[c][r]: finished columns of the factor, Xs[r][c]: finished rows of the
//   inverse, rdiag[j] = 1 / L_jj; identity past kb.
// Bound by FP64 issue (a sub-core starts a warp's FP64 instruction every 64
// cycles) and each pivot's reciprocal square root, so what is unfinished lives in
// registers (warp w: columns w, w + 8, .. with a row pair per lane, rows w, w + 8,
// .. of the inverse with a column pair per lane), one barrier a step, and the next
// column is finished while the others are updated.  Through shared memory, column
// by column, the pair took 0.158 ms; now 0.097 (the inverse alone 0.046).
template <bool FACTOR>
__device__ __forceinline__ void factor_invert(int kb, double (&L0)[8], double (&L1)[8], double (*Ls)[PB + 1],
                                              double (*Xs)[PB + 1], double* rdiag, int col0, DevStatus* st) {
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  double X0[8], X1[8];
#pragma unroll
  for (int i = 0; i < 8; i++) {
    X0[i] = wp + 8 * i == lane ? 1.0 : 0.0;
    X1[i] = wp + 8 * i == lane + 32 ? 1.0 : 0.0;
  }
  // column j of the factor from its updated values (rows lane, lane + 32)
  auto finish = [&](int j, double c0, double c1) {
    const double d = __shfl_sync(0xffffffffu, j < 32 ? c0 : c1, j & 31);
    if (!(d > 0.0) && lane == 0 && j < kb) set_status(st, FGLSGPU_ENOTSPD, col0 + j + 1, -1);
    const double ri = chain_rsqrt(d);
    double piv = d * ri;
    piv = fma(0.5 * ri, fma(-piv, piv, d), piv);
    Ls[j][lane] = lane > j ? c0 * ri : lane == j ? piv : 0.0;
    Ls[j][lane + 32] = lane + 32 > j ? c1 * ri : lane + 32 == j ? piv : 0.0;
    if (lane == 0) rdiag[j] = ri;
  };
  if (FACTOR && wp == 0) finish(0, L0[0], L1[0]);
  // j = 8 jb + j8, jb unrolled: register arrays take constant indexes only, and
  // what is finished costs nothing
#pragma unroll
  for (int jb = 0; jb < 8; jb++) {
#pragma unroll 1
    for (int j8 = 0; j8 < 8; j8++) {
      const int j = 8 * jb + j8;
      __syncthreads();
      if (FACTOR && j + 1 < PB) {
        const double l0 = -Ls[j][lane], l1 = -Ls[j][lane + 32];
        if (((j + 1) & 7) == wp) {
          const double f = Ls[j][j + 1];
          const int nx = jb < 7 ? jb + 1 : 7;
          finish(j + 1, jb < 4 ? fma(l0, f, j8 < 7 ? L0[jb] : L0[nx]) : 0.0, fma(l1, f, j8 < 7 ? L1[jb] : L1[nx]));
        }
#pragma unroll
        for (int i = jb; i < 8; i++) {
          const int c = wp + 8 * i;
          if (i <= jb + 1 && c <= j + 1) continue;
          const double f = Ls[j][c];
          if (i < 4) L0[i] = fma(l0, f, L0[i]);  // columns from 32 on have no row below 32
          L1[i] = fma(l1, f, L1[i]);
        }
      }
      if (j > 0) {  // row j - 1 of the inverse, finished a step ago, from the rows below
        const double x0 = Xs[j - 1][lane], x1 = Xs[j - 1][lane + 32];
#pragma unroll
        for (int i = jb; i < 8; i++) {
          const int r = wp + 8 * i;
          if (i == jb && r < j) continue;
          const double l = -Ls[j - 1][r];
          X0[i] = fma(l, x0, X0[i]);
          if (jb >= 4) X1[i] = fma(l, x1, X1[i]);
        }
      }
      if (j8 == wp) {
        const double rd = rdiag[j];
        Xs[j][lane] = X0[jb] * rd;
        Xs[j][lane + 32] = X1[jb] * rd;
      }
    }
  }
  __syncthreads();
}

// Factors the kb x kb diagonal block at A (lower, in place) and writes the
// inverse of its factor to dinv (PB x PB, row c at dinv + c*PB, zero above the
// diagonal and past kb).
__global__ void __launch_bounds__(DT) potf2_inv_kernel(int kb, double* A, long long lda, int col0,
                                                       double* __restrict__ dinv, DevStatus* st) {
  extern __shared__ double sm[];
  double(*Ls)[PB + 1] = (double(*)[PB + 1])sm;
  double(*Xs)[PB + 1] = (double(*)[PB + 1])(sm + PB * (PB + 1));
  __shared__ double rdiag[PB];
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  double L0[8], L1[8];
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int c = wp + 8 * i;
    const double* a = A + (long long)c * lda;
    L0[i] = (lane >= c && lane < kb) ? a[lane] : lane == c ? 1.0 : 0.0;
    L1[i] = (lane + 32 >= c && lane + 32 < kb) ? a[lane + 32] : lane + 32 == c ? 1.0 : 0.0;
  }
  factor_invert<true>(kb, L0, L1, Ls, Xs, rdiag, col0, st);
  for (int e = threadIdx.x; e < PB * PB; e += DT) {
    const int r = e & (PB - 1), c = e / PB;
    if (r >= c && r < kb) A[r + (long long)c * lda] = Ls[c][r];
    dinv[e] = (c < kb && r <= c) ? Xs[c][r] : 0.0;  // row c, element r
  }
}

// P (rows x kb) := P L^-T for the factored block, as a product with its
// inverse: 32 rows a CTA.  FP64-issue-bound: rows * kb^2 / 2 FMAs over all SMs.
__global__ void __launch_bounds__(256) panel_mul_kernel(int rows, int kb, double* __restrict__ P, long long lda,
                                                        const double* __restrict__ dinv) {
  __shared__ double Ps[PB][32], Di[PB][PB];  // Ps[q][r], Di[c][q]
  const int r = threadIdx.x & 31, cg = threadIdx.x >> 5;
  const int row = blockIdx.x * 32 + r;
  for (int e = threadIdx.x; e < PB * PB; e += 256) Di[e / PB][e & (PB - 1)] = dinv[e];
  for (int q = cg; q < PB; q += 8) Ps[q][r] = (row < rows && q < kb) ? P[row + (long long)q * lda] : 0.0;
  __syncthreads();
  double acc[8];
#pragma unroll
  for (int i = 0; i < 8; i++) acc[i] = 0.0;
#pragma unroll
  for (int qb = 0; qb < 8; qb++) {
#pragma unroll
    for (int q8 = 0; q8 < 8; q8++) {
      const double p = Ps[qb * 8 + q8][r];
#pragma unroll
      for (int i = qb; i < 8; i++) acc[i] = fma(p, Di[cg + 8 * i][qb * 8 + q8], acc[i]);  // columns cg + 8 i
    }
  }
#pragma unroll
  for (int i = 0; i < 8; i++)
    if (row < rows && cg + 8 * i < kb) P[row + (long long)(cg + 8 * i) * lda] = acc[i];
}

// Inverses of the PB x PB diagonal blocks of L, one CTA each, into Linv.
__global__ void __launch_bounds__(DT) tri_inv_kernel(int n, const double* __restrict__ L, long long ldl,
                                                     double* __restrict__ Linv) {
  extern __shared__ double sm[];
  double(*Ls)[PB + 1] = (double(*)[PB + 1])sm;
  double(*Xs)[PB + 1] = (double(*)[PB + 1])(sm + PB * (PB + 1));
  __shared__ double rdiag[PB];
  const int o = blockIdx.x * PB, kb = min(PB, n - o);
  for (int e = threadIdx.x; e < PB * PB; e += DT) {
    const int r = e & (PB - 1), c = e / PB;
    Ls[c][r] = (r >= c && r < kb) ? L[(o + r) + (long long)(o + c) * ldl] : r == c ? 1.0 : 0.0;
  }
  __syncthreads();
  if (threadIdx.x < PB) rdiag[threadIdx.x] = 1.0 / Ls[threadIdx.x][threadIdx.x];
  __syncthreads();
  double none[8];
  factor_invert<false>(kb, none, none, Ls, Xs, rdiag, 0, nullptr);
  for (int e = threadIdx.x; e < PB * PB; e += DT) {
    const int r = e & (PB - 1), c = e / PB;
    if (r >= c && r < kb && c < kb) Linv[(o + r) + (long long)(o + c) * n] = Xs[r][c];
  }
}

// Merge of neighbouring diagonal blocks [o, o + w) and [o + w, o + w + w2) of
// the inverse, o = 2 w blockIdx.z: with L21 the block of L between them,
//   FIRST:  T^T = A^-T L21^T   (into the zero block above the diagonal)
//   second: X21 = -D^-1 T
// 32 x 32 outputs a CTA; the zero halves of A^-1 and D^-1 are skipped.
template <bool FIRST>
__global__ void __launch_bounds__(256) tri_merge_kernel(int n, int w, const double* __restrict__ L, long long ldl,
                                                        double* Linv) {
  __shared__ double As[32][33], Bs[32][33];
  const int o = 2 * w * blockIdx.z, w2 = min(w, n - o - w);
  const int M = FIRST ? w : w2, N = FIRST ? w2 : w;
  const int i0 = blockIdx.x * 32, j0 = blockIdx.y * 32;
  if (w2 <= 0 || i0 >= M || j0 >= N) return;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int kbeg = FIRST ? i0 : 0, kend = FIRST ? w : min(w2, i0 + 32);
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  for (int k0 = kbeg; k0 < kend; k0 += 32) {
    __syncthreads();
    for (int q = ty; q < 32; q += 8) {
      if (FIRST) {
        // As[k][i] = A^-1(k, i): memory runs along k; Bs[k][j] = L21(j, k)
        As[tx][q] = (k0 + tx < w && i0 + q < w) ? Linv[(o + k0 + tx) + (long long)(o + i0 + q) * n] : 0.0;
        Bs[q][tx] = (j0 + tx < w2 && k0 + q < w) ? L[(o + w + j0 + tx) + (long long)(o + k0 + q) * ldl] : 0.0;
      } else {
        As[q][tx] = (i0 + tx < w2 && k0 + q < w2) ? Linv[(o + w + i0 + tx) + (long long)(o + w + k0 + q) * n] : 0.0;
        Bs[q][tx] = (j0 + tx < w && k0 + q < w2) ? Linv[(o + j0 + tx) + (long long)(o + w + k0 + q) * n] : 0.0;
      }
    }
    __syncthreads();
#pragma unroll 8
    for (int k = 0; k < 32; k++) {
      const double a = As[k][tx];
#pragma unroll
      for (int u = 0; u < 4; u++) acc[u] = fma(a, Bs[k][ty * 4 + u], acc[u]);
    }
  }
#pragma unroll
  for (int u = 0; u < 4; u++) {
    const int i = i0 + tx, j = j0 + ty * 4 + u;
    if (i >= M || j >= N) continue;
    if (FIRST) Linv[(o + i) + (long long)(o + w + j) * n] = acc[u];
    else Linv[(o + w + i) + (long long)(o + j) * n] = -acc[u];
  }
}

// Y (n x N, ld n) = Linv X: 32 rows a CTA, a row per lane, the columns of Linv up
// to the diagonal dealt to the eight warps, N <= 8 columns of X at a time.
// n^2 N / 2 FMAs and one read of the triangle (n = 6000, N = 3: 0.83 ms on 32 x 8
// tiles of the general product).
constexpr int LM = 8;
__global__ void __launch_bounds__(256) lower_mul_kernel(int n, int N, const double* __restrict__ Linv,
                                                        const double* __restrict__ X, double* __restrict__ Y) {
  __shared__ double red[8][LM][32];
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const int r0 = (gridDim.x - 1 - blockIdx.x) * 32, r = r0 + lane;  // longest rows first
  const int kend = min(n, r0 + 32);
  double acc[LM];
#pragma unroll
  for (int q = 0; q < LM; q++) acc[q] = 0.0;
#pragma unroll 4
  for (int k = wp; k < kend; k += 8) {
    const double l = r < n ? Linv[r + (long long)k * n] : 0.0;
#pragma unroll
    for (int q = 0; q < LM; q++)
      if (q < N) acc[q] = fma(l, X[k + (long long)q * n], acc[q]);
  }
#pragma unroll
  for (int q = 0; q < LM; q++) red[wp][q][lane] = acc[q];
  __syncthreads();
  if (wp < N && r < n) {
    double v = 0.0;
#pragma unroll
    for (int u = 0; u < 8; u++) v += red[u][wp][lane];
    Y[r + (long long)wp * n] = v;
  }
}
// Y (n x N, ld n) = Linv^T X: a warp per column of Linv.
__global__ void __launch_bounds__(256) lower_tmul_kernel(int n, int N, const double* __restrict__ Linv,
                                                         const double* __restrict__ X, double* __restrict__ Y) {
  const int lane = threadIdx.x & 31, j = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (j >= n) return;
  const double* l = Linv + (long long)j * n;
  double acc[LM];
#pragma unroll
  for (int q = 0; q < LM; q++) acc[q] = 0.0;
#pragma unroll 4
  for (int i = (j & ~31) + lane; i < n; i += 32) {
    const double v = l[i];  // zero above the diagonal
#pragma unroll
    for (int q = 0; q < LM; q++)
      if (q < N) acc[q] = fma(v, X[i + (long long)q * n], acc[q]);
  }
#pragma unroll
  for (int q = 0; q < LM; q++) {
    if (q >= N) break;
    double v = acc[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) Y[j + (long long)q * n] = v;
  }
}

// Zeros above the diagonal of every merged block, [o, o + w) x [o + w, ..).
__global__ void __launch_bounds__(256) tri_clear_kernel(int n, int w, double* __restrict__ Linv) {
  const int o = 2 * w * blockIdx.z, w2 = min(w, n - o - w);
  for (int e = blockIdx.x * 256 + threadIdx.x; e < w * w2; e += gridDim.x * 256)
    Linv[(o + e % w) + (long long)(o + w + e / w) * n] = 0.0;
}

// Forward substitution with the kb x kb lower block L on a set of right-hand
// sides.  RHS element (i, c) lives at X[i*si + c*sc]; i < kb runs over the
// block's rows, c < nrhs over the right-hand sides.  Used for
//   TRSM:  X := L^-1 X        (si = 1, sc = ldx)
template <int SCB>
__global__ void __launch_bounds__(DT) diag_solve_kernel(int kb, const double* L, long long ldl,
                                                        double* X, long long si, long long sc,
                                                        int nrhs) {
  constexpr int G = DT / SCB;      // row groups (a power of two)
  extern __shared__ double sm[];
  const int ldL = NB + 1;
  double* Ls = sm;                 // [NB][NB+1] column-major
  double* Xs = sm + NB * ldL;      // [SCB][NB+1]: Xs[c * ldL + i]
  const int c0 = blockIdx.x * SCB;
  const int nc = min(SCB, nrhs - c0);
  for (int e = threadIdx.x; e < kb * kb; e += DT) {
    int r = e % kb, c = e / kb;
    Ls[c * ldL + r] = (r >= c) ? L[r + (long long)c * ldl] : 0.0;
  }
  if (si == 1) {
    for (int e = threadIdx.x; e < kb * nc; e += DT) {
      int i = e % kb, c = e / kb;
      Xs[c * ldL + i] = X[i + (long long)(c0 + c) * sc];
    }
  } else {
    for (int e = threadIdx.x; e < kb * nc; e += DT) {
      int c = e % nc, i = e / nc;
      Xs[c * ldL + i] = X[(long long)i * si + (long long)(c0 + c) * sc];
    }
  }
  __syncthreads();
  const int c = threadIdx.x % SCB;   // my column
  const int g = threadIdx.x / SCB;   // my row group
  for (int j = 0; j < kb; j++) {
    double xj = 0.0;
    if (c < nc) xj = Xs[c * ldL + j] / Ls[j * ldL + j];
    __syncthreads();
    if (c < nc) {
      if (g == (j & (G - 1))) Xs[c * ldL + j] = xj;
      for (int i = j + 1 + ((g - (j + 1)) & (G - 1)); i < kb; i += G) Xs[c * ldL + i] -= Ls[j * ldL + i] * xj;
    }
    __syncthreads();
  }
  if (si == 1) {
    for (int e = threadIdx.x; e < kb * nc; e += DT) {
      int i = e % kb, cc = e / kb;
      X[i + (long long)(c0 + cc) * sc] = Xs[cc * ldL + i];
    }
  } else {
    for (int e = threadIdx.x; e < kb * nc; e += DT) {
      int cc = e % nc, i = e / nc;
      X[(long long)i * si + (long long)(c0 + cc) * sc] = Xs[cc * ldL + i];
    }
  }
}

constexpr size_t TRI_SMEM = sizeof(double) * 2 * PB * (PB + 1);  // a diagonal block and its inverse
constexpr size_t DSOLVE_SMEM = sizeof(double) * (NB + SCB) * (NB + 1);
constexpr int SCB_NARROW = 16;  // RHS per CTA when few right-hand sides (e.g. [y XL] of a trait)
constexpr size_t DSOLVE_SMEM_NARROW = sizeof(double) * (NB + SCB_NARROW) * (NB + 1);

// X := L_kk^-1 X for nrhs right-hand sides: 64 per CTA, or 16 when that
// leaves fewer CTAs than half the SMs (the solve is FP64-issue-bound per SM)
void launch_diag_solve(cudaStream_t s, int kb, const double* L, long long ldl, double* X, long long si,
                       long long sc, int nrhs) {
  if (ceil_div(nrhs, SCB) < 76)
    diag_solve_kernel<SCB_NARROW><<<ceil_div(nrhs, SCB_NARROW), DT, DSOLVE_SMEM_NARROW, s>>>(kb, L, ldl, X, si,
                                                                                           sc, nrhs);
  else
    diag_solve_kernel<SCB><<<ceil_div(nrhs, SCB), DT, DSOLVE_SMEM, s>>>(kb, L, ldl, X, si, sc, nrhs);
}

__global__ void build_shifted_kernel(int n, const double* __restrict__ S, long long lds, double alpha,
                                     double beta, double* __restrict__ A, long long lda) {
  long long total = (long long)n * n;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    int r = (int)(e % n), c = (int)(e / n);
    if (r < c) continue;
    double v = alpha * S[r + (long long)c * lds];
    if (r == c) v += beta;
    A[r + (long long)c * lda] = v;
  }
}

bool g_attr_done = false;
cudaError_t ensure_attrs() {
  if (g_attr_done) return cudaSuccess;
  FGLS_CUDA_TRY(cudaFuncSetAttribute(potf2_inv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TRI_SMEM));
  FGLS_CUDA_TRY(cudaFuncSetAttribute(tri_inv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TRI_SMEM));
  FGLS_CUDA_TRY(cudaFuncSetAttribute(diag_solve_kernel<SCB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)DSOLVE_SMEM));
  FGLS_CUDA_TRY(cudaFuncSetAttribute(diag_solve_kernel<SCB_NARROW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)DSOLVE_SMEM_NARROW));
  g_attr_done = true;
  return cudaSuccess;
}

}  // namespace

cudaError_t dgemm(cudaStream_t s, bool tA, bool tB, int M, int N, int K, double alpha,
                  const double* A, long long lda, const double* B, long long ldb, double beta,
                  double* C, long long ldc) {
  return launch_dgemm<false>(s, tA, tB, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
}

namespace {
// C = alpha * sum_z P_z + beta * C, z ascending (P_z: M x N, ld M)
__global__ void splitk_reduce_kernel(int M, int N, int splits, const double* __restrict__ P, double alpha,
                                     double beta, double* __restrict__ C, long long ldc) {
  const long long total = (long long)M * N;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    double v = 0.0;
    for (int z = 0; z < splits; z++) v += P[e + (long long)z * total];
    const int i = (int)(e % M), j = (int)(e / M);
    double* c = C + i + (long long)j * ldc;
    *c = beta != 0.0 ? fma(beta, *c, alpha * v) : alpha * v;
  }
}
}  // namespace

cudaError_t dgemm_splitk(cudaStream_t s, bool tA, bool tB, int M, int N, int K, double alpha, const double* A,
                         long long lda, const double* B, long long ldb, double beta, double* C, long long ldc,
                         double* work, long long work_elems) {
  if (M <= 0 || N <= 0) return cudaSuccess;
  const int tiles = ceil_div(M, GM) * ceil_div(N, GN);
  int splits = std::min(ceil_div(2 * 152, tiles), K / 512);
  if ((long long)M * N > 0) splits = (int)std::min<long long>(splits, work_elems / ((long long)M * N));
  if (tiles >= 152 || splits < 2 || !work)
    return launch_dgemm<false>(s, tA, tB, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
  dim3 grid(ceil_div(M, GM), ceil_div(N, GN), splits);
  if (!tA && !tB) dgemm_kernel<false, false, false><<<grid, GT, 0, s>>>(M, N, K, 1.0, A, lda, B, ldb, 0.0, work, M);
  else if (!tA && tB) dgemm_kernel<false, true, false><<<grid, GT, 0, s>>>(M, N, K, 1.0, A, lda, B, ldb, 0.0, work, M);
  else if (tA && !tB) dgemm_kernel<true, false, false><<<grid, GT, 0, s>>>(M, N, K, 1.0, A, lda, B, ldb, 0.0, work, M);
  else dgemm_kernel<true, true, false><<<grid, GT, 0, s>>>(M, N, K, 1.0, A, lda, B, ldb, 0.0, work, M);
  const long long total = (long long)M * N;
  splitk_reduce_kernel<<<(int)std::min<long long>((total + 255) / 256, 152LL * 16), 256, 0, s>>>(M, N, splits, work,
                                                                                                alpha, beta, C, ldc);
  note_launch(2);
  return cudaGetLastError();
}

cudaError_t dgemm_lower(cudaStream_t s, bool tA, bool tB, int N, int K, double alpha,
                        const double* A, long long lda, const double* B, long long ldb,
                        double beta, double* C, long long ldc) {
  return launch_dgemm<true>(s, tA, tB, N, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
}

cudaError_t build_shifted(cudaStream_t s, int n, const double* Src, long long lds, double alpha,
                          double beta, double* A, long long lda) {
  long long total = (long long)n * n;
  int blocks = (int)std::min<long long>((total + 255) / 256, 152LL * 16);
  build_shifted_kernel<<<blocks, 256, 0, s>>>(n, Src, lds, alpha, beta, A, lda);
  note_launch();
  return cudaGetLastError();
}

// Blocked Cholesky: 64-column blocks (factor and its inverse in one CTA, the
// panel below as a product with the inverse), updates within 512-column panels
// after each block and of the whole trailing triangle after each panel, so that
// the big update has K = 512.  With digits, n = 6000 takes about 22 ms.
cudaError_t dpotrf_lower(cudaStream_t s, DigitGemm* dg, int n, double* A, long long lda, double* dinv, DevStatus* st) {
  FGLS_CUDA_TRY(ensure_attrs());
  for (int k0 = 0; k0 < n; k0 += PO) {
    const int kw = std::min(PO, n - k0);
    for (int k = k0; k < k0 + kw; k += PB) {
      const int kb = std::min(PB, k0 + kw - k);
      double* Akk = A + k + (long long)k * lda;
      potf2_inv_kernel<<<1, DT, TRI_SMEM, s>>>(kb, Akk, lda, k, dinv, st);
      note_launch();
      const int rest = n - k - kb;
      if (rest <= 0) break;
      double* P = A + (k + kb) + (long long)k * lda;  // rest x kb panel
      panel_mul_kernel<<<ceil_div(rest, 32), 256, 0, s>>>(rest, kb, P, lda, dinv);
      note_launch();
      FGLS_CUDA_TRY(cudaGetLastError());
      const int in = k0 + kw - k - kb;  // columns of the panel still to factor
      if (in > 0) {
        double* T = A + (k + kb) + (long long)(k + kb) * lda;
        DigitMat a;
        if (dg && digit_gemm_pays(rest, in, kb)) a = digit_gemm_operand(dg, 0, rest, kb);
        if (a.d) {
          FGLS_CUDA_TRY(digit_cut(s, a, P, lda, false));
          DigitMat b = a;  // the panel's first rows
          b.rows = in;
          FGLS_CUDA_TRY(digit_mul(dg, s, a, b, -1.0, 1.0, T, lda));
        } else {
          FGLS_CUDA_TRY(dgemm(s, false, true, rest, in, kb, -1.0, P, lda, P, lda, 1.0, T, lda));
        }
      }
    }
    const int rest = n - k0 - kw;
    if (rest <= 0) break;
    double* P = A + (k0 + kw) + (long long)k0 * lda;  // rest x kw
    double* T = A + (k0 + kw) + (long long)(k0 + kw) * lda;
    DigitMat a;
    if (dg && digit_gemm_pays(rest, rest, kw)) a = digit_gemm_operand(dg, 0, rest, kw);
    if (a.d) {
      DigitMulOpts o;
      o.c_lower = true;
      FGLS_CUDA_TRY(digit_cut(s, a, P, lda, false));
      FGLS_CUDA_TRY(digit_mul(dg, s, a, a, -1.0, 1.0, T, lda, o));
    } else {
      FGLS_CUDA_TRY(dgemm_lower(s, false, true, rest, kw, -1.0, P, lda, P, lda, 1.0, T, lda));
    }
  }
  return cudaSuccess;
}

namespace {
// The block [off, off + size) of the inverse, its PO-blocks done: halves first,
// then X21 = -D^-1 (L21 A^-1), with T^T = A^-T L21^T in the zero block above
// the diagonal meanwhile.
cudaError_t inverse_range(cudaStream_t s, DigitGemm* dg, int n, const double* L, long long ldl, double* Linv, int off,
                          int size) {
  if (size <= PO) return cudaSuccess;
  int s1 = PO;
  while (2 * s1 < size) s1 *= 2;
  const int s2 = size - s1, o2 = off + s1;
  FGLS_CUDA_TRY(inverse_range(s, dg, n, L, ldl, Linv, off, s1));
  FGLS_CUDA_TRY(inverse_range(s, dg, n, L, ldl, Linv, o2, s2));
  double* TT = Linv + off + (long long)o2 * n;
  FGLS_CUDA_TRY(digit_dgemm(dg, s, true, true, s1, s2, s1, 1.0, Linv + off + (long long)off * n, n,
                            L + o2 + (long long)off * ldl, ldl, 0.0, TT, n));
  DigitMulOpts lower;
  lower.a_lower = true;
  FGLS_CUDA_TRY(digit_dgemm(dg, s, false, true, s2, s1, s2, -1.0, Linv + o2 + (long long)o2 * n, n, TT, n, 0.0,
                            Linv + o2 + (long long)off * n, n, lower));
  return cudaMemset2DAsync(TT, sizeof(double) * n, 0, sizeof(double) * s1, s2, s);
}
}  // namespace

// 64 x 64 blocks by substitution, all at once; neighbours merged to 512 by one
// launch a level; beyond that two products a merge, through digits.
cudaError_t lower_inverse(cudaStream_t s, DigitGemm* dg, int n, const double* L, long long ldl, double* Linv) {
  FGLS_CUDA_TRY(ensure_attrs());
  FGLS_CUDA_TRY(cudaMemsetAsync(Linv, 0, sizeof(double) * (size_t)n * n, s));
  tri_inv_kernel<<<ceil_div(n, PB), DT, TRI_SMEM, s>>>(n, L, ldl, Linv);
  note_launch();
  for (int w = PB; w < PO && w < n; w *= 2) {
    const dim3 grid(w / 32, w / 32, ceil_div(n - w, 2 * w));
    tri_merge_kernel<true><<<grid, 256, 0, s>>>(n, w, L, ldl, Linv);
    tri_merge_kernel<false><<<grid, 256, 0, s>>>(n, w, L, ldl, Linv);
    tri_clear_kernel<<<dim3(std::max(1, w * w / 2048), 1, grid.z), 256, 0, s>>>(n, w, Linv);
    note_launch(3);
  }
  FGLS_CUDA_TRY(cudaGetLastError());
  return inverse_range(s, dg, n, L, ldl, Linv, 0, n);
}

cudaError_t lower_mul(cudaStream_t s, bool trans, int n, int N, const double* Linv, const double* X, double* Y) {
  for (int q = 0; q < N; q += LM) {
    const int m = std::min(LM, N - q);
    if (trans) lower_tmul_kernel<<<ceil_div(n, 8), 256, 0, s>>>(n, m, Linv, X + (long long)q * n, Y + (long long)q * n);
    else lower_mul_kernel<<<ceil_div(n, 32), 256, 0, s>>>(n, m, Linv, X + (long long)q * n, Y + (long long)q * n);
    note_launch();
  }
  return cudaGetLastError();
}

cudaError_t dtrsm_llnn(cudaStream_t s, int n, int nrhs, const double* L, long long ldl, double* X,
                       long long ldx) {
  if (nrhs <= 0) return cudaSuccess;
  FGLS_CUDA_TRY(ensure_attrs());
  for (int k = 0; k < n; k += NB) {
    const int kb = std::min(NB, n - k);
    const double* Lkk = L + k + (long long)k * ldl;
    double* Xk = X + k;
    launch_diag_solve(s, kb, Lkk, ldl, Xk, 1, ldx, nrhs);
    note_launch();
    FGLS_CUDA_TRY(cudaGetLastError());
    const int rest = n - k - kb;
    if (rest > 0)
      FGLS_CUDA_TRY(dgemm(s, false, false, rest, nrhs, kb, -1.0, L + (k + kb) + (long long)k * ldl,
                          ldl, Xk, ldx, 1.0, X + k + kb, ldx));
  }
  return cudaSuccess;
}

}  // namespace fgls
