// Shared definitions for the GB300 FGLS engine (sm_103a).
//
// All matrices are column-major FP64 unless stated otherwise, as in the
// reference's on-disk layout (Phi n x n, XL n x wXL, XR blocks n x (x*wXR)).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "fgls_gb300.h"

namespace fgls {

// Device status word written by kernels that can fail on data (a non-SPD
// p x p system, a non-converging iteration, a bounded wait that expired).
// The first failure wins (atomicCAS on code).  Host reads it after a sync.
struct DevStatus {
  int code;      // FGLSGPU_OK or an FGLSGPU_E* code
  int info;      // LAPACK-style info (order of the failing minor, iteration count, ...)
  long long idx; // failing item (SNP index within the block, trait, row ...)
};

__device__ __forceinline__ void set_status(DevStatus* st, int code, int info, long long idx) {
  if (st && atomicCAS(&st->code, FGLSGPU_OK, code) == FGLSGPU_OK) {
    st->info = info;
    st->idx = idx;
  }
}

// 1 / sqrt(d) on a short chain: dependent FP64 instructions take some 150 cycles
// each here, and the library function is a chain of two dozen.  Seed from the FP32
// reciprocal square root of the mantissa (moved in and out by integer
// instructions), then one third-order step y (1 + e/2 + 3 e^2 / 8), e = 1 - d y^2
// (the binomial series of (1 - e)^(-1/2)): the seed's two ulps and the mantissa cut
// to 23 bits make |e| < 2^-21 + 2^-23, which leaves 5/16 |e|^3 < 2^-63.7.
__device__ __forceinline__ double chain_rsqrt(double d) {
  const long long b = __double_as_longlong(d);
  const int ex = (int)(b >> 52);
  if (ex <= 0 || ex >= 0x7ff) return rsqrt(d);  // zero, subnormal, negative, infinite, NaN
  const int k = ex - 1023, odd = k & 1;
  const float m = __int_as_float(((127 + odd) << 23) | ((int)(b >> 29) & 0x7fffff));  // in [1, 4)
  const int f = __float_as_int(rsqrtf(m));
  const double y = __longlong_as_double(((long long)((f >> 23) - 127 + 1023 - (k >> 1)) << 52) |
                                        ((long long)(f & 0x7fffff) << 29));
  const double t = d * y;
  const double e = fma(-fma(d, y, -t), y, fma(-t, y, 1.0));  // with the rounding of d y
  return fma(y * e, fma(0.375, e, 0.5), y);
}

// 1 / d on a short chain: FP32 reciprocal of the mantissa (moved in and out by
// integer instructions), then y (1 + e + e^2), e = 1 - d y (the geometric series of
// 1 / (1 - e)); |e| < 2^-22 leaves 2^-66.
__device__ __forceinline__ double chain_rcp(double d) {
  const long long b = __double_as_longlong(d);
  const int ex = (int)(b >> 52) & 0x7ff;
  if (ex <= 1 || ex >= 0x7fd) return 1.0 / d;
  const int f = __float_as_int(__frcp_rn(__int_as_float(0x3f800000 | ((int)(b >> 29) & 0x7fffff))));  // in [0.5, 1]
  const double y = __longlong_as_double(((long long)((f >> 23) - 127 - (ex - 1023) + 1023) << 52) |
                                        ((long long)(f & 0x7fffff) << 29) | (b & (long long)0x8000000000000000ull));
  const double e = fma(-d, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

inline int ceil_div(long long a, long long b) { return (int)((a + b - 1) / b); }

// The engines of this process on the current device that are between calls give back
// the memory that only makes them faster (fgls_engine.cu); false if none holds any.
bool engines_give_back();
// Device memory that a call outside of an engine cannot do without.
template <class T>
cudaError_t needed_malloc(T** p, size_t bytes) {
  cudaError_t r = cudaMalloc((void**)p, bytes);
  if (r == cudaErrorMemoryAllocation) {
    (void)cudaGetLastError();
    if (engines_give_back()) r = cudaMalloc((void**)p, bytes);
  }
  return r;
}

// Kernel launchers (host side, defined in the .cu files).  All are
// asynchronous on `s` and return cudaError_t of the launch.

// C = alpha * op(A) * op(B) + beta * C   (FP64, column-major, op = N or T)
cudaError_t dgemm(cudaStream_t s, bool transA, bool transB, int M, int N, int K, double alpha,
                  const double* A, long long lda, const double* B, long long ldb, double beta,
                  double* C, long long ldc);
// The same product with K split over CTAs when M x N has too few 64 x 64
// tiles to fill the GPU (partials in work, work_elems doubles, then summed in
// a fixed order); falls back to dgemm when splitting does not apply.
cudaError_t dgemm_splitk(cudaStream_t s, bool transA, bool transB, int M, int N, int K, double alpha,
                         const double* A, long long lda, const double* B, long long ldb, double beta, double* C,
                         long long ldc, double* work, long long work_elems);
// Lower-triangle-only variant (C n x n lower, tiles strictly above the
// diagonal are skipped; entries above the diagonal inside diagonal tiles
// are written too and must be ignored by the caller).
cudaError_t dgemm_lower(cudaStream_t s, bool transA, bool transB, int N, int K, double alpha,
                        const double* A, long long lda, const double* B, long long ldb,
                        double beta, double* C, long long ldc);

// In-place lower Cholesky of the n x n matrix A (only the lower triangle is
// read; the strict upper triangle is scratch).  dg (may be null): the trailing
// updates run as exact digit products (fgls_digit_gemm.cuh); dinv: scratch of
// 64 x 64.  Returns cudaSuccess or a launch error; a non-positive pivot is
// reported through `st` (info = 1-based column).
struct DigitGemm;
cudaError_t dpotrf_lower(cudaStream_t s, DigitGemm* dg, int n, double* A, long long lda, double* dinv, DevStatus* st);
// Linv = L^-1 (n x n, ld n, zero above the diagonal) of the lower triangle of L.
cudaError_t lower_inverse(cudaStream_t s, DigitGemm* dg, int n, const double* L, long long ldl, double* Linv);
// Y = Linv X or Linv^T X for few columns (n x N, ld n; Y must not be X).
cudaError_t lower_mul(cudaStream_t s, bool trans, int n, int N, const double* Linv, const double* X, double* Y);
cudaError_t build_shifted(cudaStream_t s, int n, const double* Src, long long lds, double alpha,
                          double beta, double* A, long long lda);

// X := L^{-1} X   (L n x n lower, non-unit; X n x nrhs).  Blocked: diagonal
// blocks solved in shared memory, off-diagonal updates through dgemm.
cudaError_t dtrsm_llnn(cudaStream_t s, int n, int nrhs, const double* L, long long ldl, double* X,
                       long long ldx);

}  // namespace fgls

#define FGLS_CUDA_TRY(expr)                                  \
  do {                                                       \
    cudaError_t _e = (expr);                                 \
    if (_e != cudaSuccess) return _e;                        \
  } while (0)
