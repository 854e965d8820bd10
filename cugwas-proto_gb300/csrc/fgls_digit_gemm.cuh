// FP64 matrix products on the FP8 tensor cores (fgls_digit_gemm.cu): both
// operands are cut into twelve signed base-32 digits per row (60 bits under a
// power-of-two scale per row) and the digit products are summed exactly.  The
// error is normwise: below K 2^-58 2^exA 2^exB of the row scales (each between two
// and four times the row's largest element) and one rounding, where an FP64 DGEMM's
// is relative to sum |a||b|.  For rows whose elements are of one size that is the
// smaller of the two; an element 2^-k of its row's largest keeps 60 - k bits, and
// none from k = 60 on, so rows of mixed magnitude against rows mixed the other way
// belong on the FP64 kernels (row (2^70, 1) by column (0, 1): 0 instead of 1).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace fgls {

constexpr int DG_DIGITS = 12;

// One operand as digits: `rows` rows (rows of op(A), columns of op(B)) of K
// digits each, K innermost, rows of Kpad bytes, digit planes one after the
// other; per row the exponent of its scale, per 256 rows the digits in use.
struct DigitMat {
  uint8_t* d = nullptr;
  int* ex = nullptr;
  int* nd = nullptr;
  int rows = 0, K = 0, Kpad = 0;
  int prow = 0;  // rows between digit planes (rows, more in a view of the first rows)
};
size_t digit_mat_bytes(int rows, int K);
// lays out a matrix of `rows` x K in `mem` (digit_mat_bytes, 256-byte aligned)
DigitMat digit_mat_at(void* mem, int rows, int K);

// Digits of a column-major FP64 matrix.  kcontig: row r's element k at
// X[k + r*ld]; else at X[r + k*ld].  A row that holds a NaN or an infinity makes every
// product with it NaN, but infinite where its non-finite elements are infinities of one
// sign (kcontig only) and the other row was cut by digit_cut_signed and is of one sign.
cudaError_t digit_cut(cudaStream_t s, const DigitMat& m, const double* X, long long ld, bool kcontig);
cudaError_t digit_cut_signed(cudaStream_t s, const DigitMat& m, const double* X, long long ld);  // contiguous in K
// rows r = (i*w + c)*w + d: the products of columns i*w + c and i*w + d of X
cudaError_t digit_cut_products(cudaStream_t s, const DigitMat& m, const double* X, long long ld, int w);

// Workspace of the digit GEMM for one stream at a time: partial sums of every
// CTA, K-split partials, the operands of digit_dgemm, a wait error word.
struct DigitGemm;
cudaError_t digit_gemm_create(DigitGemm** out);  // cudaErrorNotSupported: no clusters of two
// Takes the partial sums' memory (120 MB), which no product is run without; digit_dgemm
// and the operands below do it themselves.  False when the device has not the memory.
bool digit_gemm_ready(DigitGemm* g);
void digit_gemm_destroy(DigitGemm* g);
int* digit_gemm_error_word(DigitGemm* g);
// whether products were launched since the word was last read (digit_gemm_checked)
bool digit_gemm_unchecked(const DigitGemm* g);
void digit_gemm_checked(DigitGemm* g);
// limit of one wait of the products launched from now on (0: the default, 2 s)
void digit_gemm_set_wait_limit(DigitGemm* g, unsigned long long ns);

struct DigitMulOpts {
  bool a_lower = false;    // row r of A is zero beyond column r
  bool c_lower = false;    // square C: only r >= c is computed and written
};
// C (A.rows x B.rows, ld ldc) = alpha * A * B^T + beta * C; A.K == B.K.
cudaError_t digit_mul(DigitGemm* g, cudaStream_t s, const DigitMat& A, const DigitMat& B, double alpha, double beta,
                      double* C, long long ldc, const DigitMulOpts& o = DigitMulOpts());

// As dgemm (fgls_common.cuh), through digits when the product is large enough
// for that to pay and `g` is set, else the FP64 kernel.  Both operands' digits
// live in g (grown on demand; without the memory for it the FP64 kernel runs).
cudaError_t digit_dgemm(DigitGemm* g, cudaStream_t s, bool tA, bool tB, int M, int N, int K, double alpha,
                        const double* A, long long lda, const double* B, long long ldb, double beta, double* C,
                        long long ldc, const DigitMulOpts& o = DigitMulOpts());
// scratch operands of g (0, 1) laid out for rows x K; d == nullptr when the
// device has not the memory
DigitMat digit_gemm_operand(DigitGemm* g, int q, int rows, int K);
// room for operands of up to `rows` x K each (so that digit_dgemm allocates
// nothing); false when the device has not the memory.  digit_gemm_trim gives
// the operands' room back, digit_gemm_release that of the partial sums too.
bool digit_gemm_reserve(DigitGemm* g, int rows, int K);
bool digit_gemm_trim(DigitGemm* g);
bool digit_gemm_release(DigitGemm* g);
// whether digit_dgemm takes the digits for this product
bool digit_gemm_pays(long long M, long long N, long long K);

}  // namespace fgls
