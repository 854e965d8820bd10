// FP64 dense kernels for the plain (all-FP64) path: tiled DGEMM, blocked
// lower Cholesky (the reference's dpotrf of M, src/fgls_chol.c:252-271) and
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

template <bool LOWER>
cudaError_t launch_dgemm(cudaStream_t s, bool tA, bool tB, int M, int N, int K, double alpha,
                         const double* A, long long lda, const double* B, long long ldb,
                         double beta, double* C, long long ldc) {
  if (M <= 0 || N <= 0) return cudaSuccess;
  dim3 grid(ceil_div(M, GM), ceil_div(N, GN));
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

// Inverse of the kb x kb lower triangle in Ls ([c][r], rdiag[j] = 1 / L_jj) into
// Xs ([c][r], zero above the diagonal): thread (c, g) holds column c's rows g,
// g + 4, ..; all threads of the CTA call it.
__device__ __forceinline__ void tri_inverse(int kb, const double (*Ls)[PB + 1], const double* rdiag,
                                            double (*Xs)[PB + 1]) {
  const int c = threadIdx.x & (PB - 1), g = threadIdx.x / PB;
  for (int r = g; r < PB; r += DT / PB) Xs[c][r] = r == c ? 1.0 : 0.0;
  __syncthreads();
  for (int j = 0; j < kb; j++) {
    const double x = Xs[c][j] * rdiag[j];
    __syncthreads();
    if (g == (j & 3)) Xs[c][j] = x;
    if (c <= j)
      for (int r = j + 1 + ((g - (j + 1)) & 3); r < kb; r += 4) Xs[c][r] = fma(-Ls[j][r], x, Xs[c][r]);
    __syncthreads();
  }
}

// Factors the kb x kb diagonal block at A (lower, in place) and writes the
// inverse of its factor to dinv (PB x PB, row c at dinv + c*PB, zero above the
// diagonal and past kb).  One CTA, a serial chain of 2 kb steps: 64 columns
// take 0.04 ms; the 128-column form was bound by one SM's FP64 rate.
__global__ void __launch_bounds__(DT) potf2_inv_kernel(int kb, double* A, long long lda, int col0,
                                                       double* __restrict__ dinv, DevStatus* st) {
  extern __shared__ double sm[];
  double(*Ls)[PB + 1] = (double(*)[PB + 1])sm;              // Ls[c][r] = A(r, c)
  double(*Xs)[PB + 1] = (double(*)[PB + 1])(sm + PB * (PB + 1));
  __shared__ double rdiag[PB];
  for (int e = threadIdx.x; e < PB * PB; e += DT) {
    const int r = e & (PB - 1), c = e / PB;
    Ls[c][r] = (r >= c && r < kb) ? A[r + (long long)c * lda] : 0.0;
  }
  __syncthreads();
  const int r = threadIdx.x & (PB - 1), g = threadIdx.x / PB;
  bool bad = false;
  for (int j = 0; j < kb; j++) {
    const double d = Ls[j][j];
    if (!(d > 0.0) && threadIdx.x == 0 && !bad) {
      bad = true;
      set_status(st, FGLSGPU_ENOTSPD, col0 + j + 1, -1);
    }
    const double piv = sqrt(d), ri = 1.0 / piv;
    const double v = r > j ? Ls[j][r] * ri : r == j ? piv : 0.0;
    __syncthreads();
    if (g == 0 && r >= j) Ls[j][r] = v;
    if (threadIdx.x == 0) rdiag[j] = ri;
    __syncthreads();
    // columns c > j of row r (the factor's column j in shared memory)
    for (int c = j + 1 + ((g - (j + 1)) & 3); c <= r; c += DT / PB) Ls[c][r] = fma(-v, Ls[j][c], Ls[c][r]);
    __syncthreads();
  }
  tri_inverse(kb, Ls, rdiag, Xs);
  for (int e = threadIdx.x; e < PB * PB; e += DT) {
    const int rr = e & (PB - 1), c = e / PB;
    if (rr >= c && rr < kb) A[rr + (long long)c * lda] = Ls[c][rr];
    // row c' = e / PB of dinv, element q = e % PB: Linv(c', q)
    dinv[e] = (c < kb && rr <= c) ? Xs[rr][c] : 0.0;
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
    Ls[c][r] = (r >= c && r < kb) ? L[(o + r) + (long long)(o + c) * ldl] : 0.0;
  }
  __syncthreads();
  if (threadIdx.x < kb) rdiag[threadIdx.x] = 1.0 / Ls[threadIdx.x][threadIdx.x];
  __syncthreads();
  tri_inverse(kb, Ls, rdiag, Xs);
  for (int e = threadIdx.x; e < PB * PB; e += DT) {
    const int r = e & (PB - 1), c = e / PB;
    if (r >= c && r < kb && c < kb) Linv[(o + r) + (long long)(o + c) * n] = Xs[c][r];
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
constexpr int SCB_NARROW = 16;  // RHS per CTA when few right-hand sides (e.g. the 512-wide L^-1 panels)
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
// the big update has K = 512.  With digits, n = 10000 takes ~30 ms against
// 360 ms when every update ran on the FP64 kernel.
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
