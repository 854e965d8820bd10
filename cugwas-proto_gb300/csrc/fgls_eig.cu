// FP64 symmetric eigendecomposition Phi = Z diag(W) Z^T on the device,
// replacing the reference's one-off dsyevr('V','A','L') (src/fgls_eigen.c:
// 861-893).  W ascending, Z orthonormal columns.
//
// Algorithm (all FP64, no vendor library):
//  1. Householder reduction to tridiagonal form in panels of 64 columns (the
//     scheme of LAPACK's dsytrd/dlatrd): within a panel a column is brought up to
//     date from the panel's V and W, and A v runs over the trailing matrix as it
//     was at the panel's start; then A -= V W^T + W V^T in one product of K = 128.
//     A is kept in full storage, so that A v is one contiguous dot product per
//     column; its power-of-two scale keeps V and W of one size (the product cuts
//     rows of [V W] into digits under one scale).
//  2. Eigenpairs of the tridiagonal by divide and conquer (fgls_dc.cu):
//     eigenvalues ascending, eigenvectors V of T.
//  3. Z = H_0 H_1 ... H_{n-3} V applied in blocks of 512 reflectors in
//     compact-WY form (Y, T from tau and Y^T Y): products only.
#include <algorithm>
#include <cfloat>
#include <cstdio>
#include <cstdlib>

#include "fgls_common.cuh"
#include "fgls_digit_gemm.cuh"
#include "fgls_kernels.cuh"

namespace fgls {

namespace {

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Largest |element| of the lower triangle, as the bits of a non-negative double
// (ordered like integers; a NaN or an infinity is the largest), into *top.
__global__ void __launch_bounds__(256) lower_max_kernel(int n, const double* __restrict__ A, long long lda,
                                                        unsigned long long* __restrict__ top) {
  unsigned long long m = 0;
  for (int c = blockIdx.x; c < n; c += gridDim.x)
    for (int r = c + threadIdx.x; r < n; r += 256)
      m = max(m, (unsigned long long)__double_as_longlong(A[r + (long long)c * lda]) & 0x7fffffffffffffffull);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(top, m);
}
// Exponent of the power of two that brings the largest element to about
// 1 / sqrt(n), so that the largest eigenvalue lies in about [1 / sqrt(n), sqrt(n)];
// 0 where there is none.
__device__ __forceinline__ int norm_shift(int n, unsigned long long top) {
  const int ex = (int)(top >> 52);
  return ex == 0 || ex == 0x7ff ? 0 : 1023 - ex - (31 - __clz(n)) / 2;
}

// A := the symmetric matrix of Src's lower triangle times 2^norm_shift, full
// storage, 32 x 32 tiles turned in shared memory (src == dst allowed: the mirror
// image of the lower triangle, unscaled with top == nullptr).
__global__ void __launch_bounds__(256) symmetrize_kernel(int n, const double* Src, long long lds, double* A,
                                                         long long lda, const unsigned long long* __restrict__ top) {
  if (blockIdx.x < blockIdx.y) return;
  __shared__ double t[32][33];
  const int r0 = blockIdx.x * 32, c0 = blockIdx.y * 32, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int sh = top ? norm_shift(n, *top) : 0;
  for (int c = ty; c < 32; c += 8) {
    const int r = r0 + tx, cc = c0 + c;
    if (r < n && cc < n && r >= cc) {
      double v = Src[r + (long long)cc * lds];
      if (sh) v = ldexp(v, sh);
      t[c][tx] = v;
      if (top) A[r + (long long)cc * lda] = v;
    }
  }
  __syncthreads();
  for (int c = ty; c < 32; c += 8) {
    const int r = c0 + tx, cc = r0 + c;  // row of the upper triangle
    if (r < n && cc < n && cc > r) A[r + (long long)cc * lda] = t[tx][c];
  }
}
__global__ void unscale_kernel(int n, double* W, const unsigned long long* __restrict__ top) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) W[i] = ldexp(W[i], -norm_shift(n, *top));
}

// Scalars of the Householder reflector of x (x[0] = alpha, |x[1:]|^2 = xnorm2):
// beta, tau and the scale of x[1:] into v[1:].
__device__ __forceinline__ void reflector(double alpha, double xnorm2, double& beta, double& tau, double& scal) {
  if (xnorm2 == 0.0) {
    tau = 0.0;
    beta = alpha;
    scal = 0.0;
  } else {
    beta = -copysign(sqrt(alpha * alpha + xnorm2), alpha);
    tau = (beta - alpha) / beta;
    scal = 1.0 / (alpha - beta);
  }
}

// Panel of columns k0 .. k0 + TB - 1: P = [V W V] (n x 3 TB, ld n), column q of V
// the reflector of column k0 + q (1 at row k0 + q + 1, zero above), W the vectors
// of the rank-2 updates.  Two launches a column:
//   tridiag_col   column i - 1's w from y = A v and the dot products of v with V
//                 and W, then column i of A brought up to date
//   tridiag_mv    the reflector of that column (every CTA derives the same
//                 scalars), y = A v, t = [W^T v ; V^T v] and the parts of y^T v
// Sums over CTAs are taken from arrays of parts in a fixed order.
constexpr int TB = 64;
// Both kernels may be launched before the one ahead of them ends (programmatic
// dependent launch): a column's two launches are on the chain of 2 n of them.  What
// that one writes changes while they run, so none of their pointers is declared
// constant or unaliased: the compiler could then read ahead of the wait.
__device__ __forceinline__ void launch_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

constexpr int TR = 32;  // rows per CTA of tridiag_col, one per lane; the panel's columns are dealt to the warps

// Panel column i = k - k0.  pend: w of column i - 1 is due,
//   w = tau (y - V t1 - W t2) + g v,  g = -tau/2 p^T v,  p^T v = tau (y^T v - 2 t1 . t2)
// (p the bracket times tau; V, W the columns before i - 1).  live: column k is
// wanted, x_r = A[r, k] - sum_q V[r, q] W[k, q] + W[r, q] V[k, q]; x_k is d[k],
// and the parts of |x[k+2:]|^2 go to npart.
__global__ void __launch_bounds__(256) tridiag_col_kernel(int n, int k, int i, bool pend, bool live,
                                                          double* A, long long lda, double* P, double* y, double* t,
                                                          double* yvpart, int nyv, double* tau, double* d, double* x,
                                                          double* npart) {
  __shared__ double st1[TB], st2[TB], vk[TB], wk[TB], part[2][8][TR], yvs[8], wsum;
  const int q1 = pend ? i - 1 : 0;  // panel columns that are complete
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const int r = k + blockIdx.x * TR + lane;
  const double *V = P, *W = P + (long long)TB * n;
  double yr = 0.0, vr = 0.0, ar = 0.0, tk = 0.0, yk = 0.0;  // what the last part needs, in flight early
  wait_previous();
  if (wp == 0 && r < n) {
    if (live) ar = A[r + (long long)k * lda];
    if (pend) {
      yr = y[r];
      vr = V[r + (long long)q1 * n];
    }
  }
  if (pend) {
    tk = tau[k - 1];
    yk = y[k];
    if (threadIdx.x < q1) {
      st1[threadIdx.x] = t[threadIdx.x];
      st2[threadIdx.x] = t[TB + threadIdx.x];
      vk[threadIdx.x] = V[k + (long long)threadIdx.x * n];
      wk[threadIdx.x] = W[k + (long long)threadIdx.x * n];
    }
    double yv = 0.0;
    for (int c = threadIdx.x; c < nyv; c += 256) yv += yvpart[c];
    __syncthreads();
    if (threadIdx.x < q1) yv = fma(-2.0 * st1[threadIdx.x], st2[threadIdx.x], yv);
    double a1 = 0.0, a2 = 0.0;
    if (r < n) {
#pragma unroll
      for (int u = 0; u < TB / 8; u++) {
        const int q = wp + 8 * u;
        if (q >= q1) break;
        const double v = V[r + (long long)q * n], w = W[r + (long long)q * n];
        a1 = fma(v, st1[q], fma(w, st2[q], a1));
        a2 = fma(v, wk[q], fma(w, vk[q], a2));
      }
    }
    part[0][wp][lane] = a1;
    part[1][wp][lane] = a2;
    yv = warp_sum(yv);
    if (lane == 0) yvs[wp] = yv;
    if (wp == 7) {  // the bracket's sum for row k, whose w every row's update needs
      double a = 0.0;
      for (int q = lane; q < q1; q += 32) a = fma(vk[q], st1[q], fma(wk[q], st2[q], a));
      a = warp_sum(a);
      if (lane == 0) wsum = a;
    }
    __syncthreads();
  }
  launch_next();
  if (wp > 0) return;
  double sq = 0.0, xr = ar;
  if (pend) {
    double a1 = 0.0, a2 = 0.0, yv = 0.0;
#pragma unroll
    for (int u = 0; u < 8; u++) {
      a1 += part[0][u][lane];
      a2 += part[1][u][lane];
      yv += yvs[u];
    }
    const double g = -0.5 * tk * tk * yv;
    const double wlast = fma(tk, yk - wsum, g);  // v_k = 1
    const double w = fma(tk, yr - a1, g * vr);
    if (r < n) P[r + (long long)(TB + q1) * n] = w;
    xr -= a2 + fma(vr, wlast, w);
  }
  if (!live) return;
  if (r < n) {
    if (r == k) d[k] = xr;
    else x[r] = xr;
    if (r >= k + 2) sq = xr * xr;
  }
  sq = warp_sum(sq);
  if (lane == 0) npart[blockIdx.x] = sq;
}

// y = A22 v, t = [W^T v ; V^T v] over rows and columns k+1 .. (i complete panel
// columns), a warp per column, and the parts of y^T v.  v = scal x below its
// leading 1, so the dot products run on x at once and take the scale at the end;
// the ninth warp derives the reflector meanwhile.  Bound by the m^2 FP64 FMAs (an
// SM takes a warp's in 16 cycles: 20 us at m = 3500) and, below m of about 1500,
// by latency.
constexpr int MV_THREADS = 288;
__global__ void __launch_bounds__(MV_THREADS) tridiag_mv_kernel(int n, int k, int i, double* A, long long lda, double* P,
                                                                double* x, double* npart, int nnp, double* tau_out,
                                                                double* e_out, double* y, double* t, double* yvpart) {
  __shared__ double sscal, yvs[8];
  const int m = n - k - 1, r0 = k + 1;
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const int warps = gridDim.x * 8, cols = m + 2 * i;
  const double* xs = x + r0;
  auto column = [&](int j) -> const double* {
    return j < m ? A + r0 + (long long)(r0 + j) * lda
                 : j < m + i ? P + r0 + (long long)(TB + j - m) * n : P + r0 + (long long)(j - m - i) * n;
  };
  auto dot = [&](int j) -> double {  // x[1:] with the column, every lane
    const double* a = column(j);
    double s0 = 0.0, s1 = 0.0;
    int r = lane;
    if (lane == 0) r = 32;  // row 0 goes in apart
#pragma unroll 4
    for (; r + 32 < m; r += 64) {
      s0 = fma(a[r], xs[r], s0);
      s1 = fma(a[r + 32], xs[r + 32], s1);
    }
    if (r < m) s0 = fma(a[r], xs[r], s0);
    return warp_sum(s0 + s1);
  };
  const int j0 = blockIdx.x * 8 + wp;
  double first = 0.0, head = 0.0;
  wait_previous();
  if (wp < 8) {
    if (j0 < cols) {
      head = column(j0)[0];
      first = dot(j0);
    }
  } else {
    double xn2 = 0.0;
    for (int c = lane; c < nnp; c += 32) xn2 += npart[c];
    xn2 = warp_sum(xn2);
    double beta, tau, scal;
    reflector(xs[0], xn2, beta, tau, scal);
    if (lane == 0) sscal = scal;
    if (blockIdx.x == 0 && lane == 0) {
      tau_out[k] = tau;
      e_out[k] = beta;
    }
  }
  __syncthreads();
  const double scal = sscal;
  // the reflector: the panel's two copies and column k of A (for the back-transform)
  for (int j = blockIdx.x * MV_THREADS + threadIdx.x; j < m + i + 1; j += gridDim.x * MV_THREADS) {
    const int r = k - i + j;
    const double v = r < r0 ? 0.0 : r == r0 ? 1.0 : x[r] * scal;
    P[r + (long long)i * n] = v;
    P[r + (long long)(2 * TB + i) * n] = v;
    if (r > r0) A[r + (long long)k * lda] = v;
  }
  if (wp == 8) {
    launch_next();
    return;
  }
  double yv = 0.0;
  for (int j = j0; j < cols; j += warps) {
    if (j != j0) {
      head = column(j)[0];
      first = dot(j);
    }
    const double s = fma(scal, first, head);
    if (lane == 0) {
      if (j < m) {
        y[r0 + j] = s;
        yv = fma(s, j == 0 ? 1.0 : xs[j] * scal, yv);
      } else {
        t[j < m + i ? j - m : TB + j - m - i] = s;
      }
    }
  }
  launch_next();
  if (lane == 0) yvs[wp] = yv;
  asm volatile("bar.sync 1, 256;" ::: "memory");  // the eight column warps
  if (threadIdx.x == 0) {
    double v = 0.0;
#pragma unroll
    for (int u = 0; u < 8; u++) v += yvs[u];
    yvpart[blockIdx.x] = v;
  }
}
constexpr int EIG_CTAS = 608;  // most CTAs of tridiag_mv: four an SM

// The last 2 x 2 block.
__global__ void tridiag_tail_kernel(int n, const double* A, long long lda, double* d, double* e) {
  if (n >= 2) {
    d[n - 2] = A[(n - 2) + (long long)(n - 2) * lda];
    e[n - 2] = A[(n - 1) + (long long)(n - 2) * lda];
  }
  d[n - 1] = A[(n - 1) + (long long)(n - 1) * lda];
  e[n - 1] = 0.0;
}

template <class... P, class... T>
cudaError_t launch_chained(void (*kernel)(P...), int grid, int block, cudaStream_t s, T... args) {
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

int grid_for(long long total) { return (int)std::min<long long>((total + 255) / 256, 152LL * 32); }

// Y (mr x nb, ld mr): reflectors b .. b+nb-1 as explicit columns over rows
// b+1 .. n-1: column c is zero above row c, 1 at row c, A[b+c+1+i, b+c] below.
__global__ void build_y_kernel(int n, int b, int nb, const double* __restrict__ A, long long lda,
                               double* __restrict__ Y) {
  const int mr = n - b - 1;
  const long long total = (long long)mr * nb;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(e % mr), c = (int)(e / mr);
    double v = 0.0;
    if (r == c) v = 1.0;
    else if (r > c) v = A[(b + 1 + r) + (long long)(b + c) * lda];
    Y[e] = v;
  }
}

// Compact-WY factor T (nb x nb upper, ld nb) of H_b ... H_{b+nb-1} =
// I - Y T Y^T from tau and G = Y^T Y (forward, columnwise):
//   T_ii = tau_i, T[0:i, i] = -tau_i T[0:i, 0:i] G[0:i, i].
// Column by column that is one CTA's serial chain through global memory (2.0
// ms at nb = 256).  Instead 32 x 32 diagonal blocks, one warp each, then
// merges of neighbours, [T1, -T1 G12 T2; 0, T2], 32 -> 64 -> .. with one
// thread per element and 16 x 16 outputs per CTA: seven launches, 0.05 ms.
constexpr int LB = 32;
__global__ void __launch_bounds__(LB) larft_base_kernel(int nb, const double* __restrict__ tau,
                                                        const double* __restrict__ G, double* __restrict__ T) {
  __shared__ double g[LB][LB + 1], t[LB][LB + 1];  // [column][row]
  const int o = blockIdx.x * LB, m = min(LB, nb - o), r = threadIdx.x;
  for (int i = 0; i < m; i++) {
    g[i][r] = r < i ? G[(o + r) + (long long)(o + i) * nb] : 0.0;
    t[i][r] = 0.0;
  }
  __syncwarp();
  for (int i = 0; i < m; i++) {
    const double ti = tau[o + i];
    double acc = 0.0;
    for (int q = r; q < i; q++) acc = fma(t[q][r], g[i][q], acc);
    if (r < i) t[i][r] = -ti * acc;
    if (r == i) t[i][r] = ti;
    __syncwarp();
  }
  for (int i = 0; i < m; i++)
    if (r < m) T[(o + r) + (long long)(o + i) * nb] = t[i][r];
}
// Merge of the blocks [o, o + w) and [o + w, o + w + w2), o = 2 w blockIdx.z:
// first P = G12 T2, then T12 = -T1 P.
template <bool FIRST>
__global__ void __launch_bounds__(256) larft_merge_kernel(int nb, int w, const double* __restrict__ G,
                                                          double* __restrict__ T, double* __restrict__ P) {
  const int o = 2 * w * blockIdx.z, w2 = min(w, nb - o - w);
  const int r = blockIdx.x * 16 + (threadIdx.x & 15), c = blockIdx.y * 16 + (threadIdx.x >> 4);
  if (r >= w || c >= w2) return;
  double* p = P + (long long)blockIdx.z * w * w;
  double acc = 0.0;
  if (FIRST) {
    for (int q = 0; q <= c; q++)
      acc = fma(G[(o + r) + (long long)(o + w + q) * nb], T[(o + w + q) + (long long)(o + w + c) * nb], acc);
    p[r + c * w] = acc;
  } else {
    for (int q = r; q < w; q++) acc = fma(T[(o + r) + (long long)(o + q) * nb], p[q + c * w], acc);
    T[(o + r) + (long long)(o + w + c) * nb] = -acc;
  }
}
// T from G and tau; P: scratch of nb^2 / 2 elements
cudaError_t larft(cudaStream_t s, int nb, const double* tau, const double* G, double* T, double* P, long long* nl) {
  FGLS_CUDA_TRY(cudaMemsetAsync(T, 0, sizeof(double) * nb * nb, s));
  larft_base_kernel<<<ceil_div(nb, LB), LB, 0, s>>>(nb, tau, G, T);
  (*nl)++;
  for (int w = LB; w < nb; w *= 2) {
    const dim3 grid(ceil_div(w, 16), ceil_div(w, 16), ceil_div(nb - w, 2 * w));
    larft_merge_kernel<true><<<grid, 256, 0, s>>>(nb, w, G, T, P);
    larft_merge_kernel<false><<<grid, 256, 0, s>>>(nb, w, G, T, P);
    *nl += 2;
  }
  return cudaGetLastError();
}

}  // namespace

size_t eig_workspace_bytes(int n) {
  // d, e, tau, x, y (n each), t (2 TB), parts of the column norm (n / TR) and of
  // y^T v (up to EIG_CTAS), the panel (n x 3 TB), the norm and the failure flag
  return sizeof(double) * ((size_t)n * (5 + 3 * TB) + 2 * TB + (n + TR - 1) / TR + 2 + EIG_CTAS + 2) + 256;
}

cudaError_t dsyev_device(cudaStream_t s, DigitGemm* dg, int n, const double* Phi, long long ldp, double* A, double* Z,
                         double* W, void* work, int* fail_out, long long* launches) {
  double* d = (double*)work;
  double* e = d + n;
  double* tau = e + n;
  double* xb = tau + n;                             // the current column
  double* yb = xb + n;                              // A v
  double* tb = yb + n;                              // W^T v, V^T v
  double* npart = tb + 2 * TB;                      // parts of the column's sum of squares
  double* yvpart = npart + (n + TR - 1) / TR + 2;   // parts of y^T v
  double* P = yvpart + EIG_CTAS;                    // [V W V]
  unsigned long long* top = (unsigned long long*)(P + (size_t)n * 3 * TB);
  int* dfail = (int*)(top + 1);
  long long nl = 0;
  // FGLS_EIG_TIMING=1 prints the phase times (CUDA events on s) to stderr
  const bool timing = getenv("FGLS_EIG_TIMING") != nullptr;
  cudaEvent_t ev[5];
  if (timing)
    for (auto& x : ev) cudaEventCreate(&x);
  auto mark = [&](int i) {
    if (timing) cudaEventRecord(ev[i], s);
  };
  // the products' digits: largest operands n x n; given back below
  if (dg && !(digit_gemm_pays(n, n, 256) && digit_gemm_reserve(dg, n, n))) {
    digit_gemm_trim(dg);
    dg = nullptr;
  }
  mark(0);
  // A := Phi's lower triangle, scaled, in full storage
  FGLS_CUDA_TRY(cudaMemsetAsync(top, 0, sizeof(*top), s));
  lower_max_kernel<<<std::min(n, 1216), 256, 0, s>>>(n, Phi, ldp, top);
  const dim3 tiles(ceil_div(n, 32), ceil_div(n, 32));
  symmetrize_kernel<<<tiles, 256, 0, s>>>(n, Phi, ldp, A, n, top);
  nl += 2;
  FGLS_CUDA_TRY(cudaGetLastError());
  // 1. tridiagonalization
  for (int k0 = 0; k0 + 2 < n; k0 += TB) {
    const int nb = std::min(TB, n - 2 - k0);
    int nyv = 0;
    for (int i = 0; i < nb; i++) {
      const int k = k0 + i, m = n - k - 1;
      const int nr = ceil_div(n - k, TR);
      FGLS_CUDA_TRY(launch_chained(tridiag_col_kernel, nr, 256, s, n, k, i, i > 0, true, A, (long long)n, P, yb, tb,
                                   yvpart, nyv, tau, d, xb, npart));
      nyv = std::min(ceil_div(m + 2 * i, 8), EIG_CTAS);
      FGLS_CUDA_TRY(launch_chained(tridiag_mv_kernel, nyv, MV_THREADS, s, n, k, i, A, (long long)n, P, xb, npart, nr,
                                   tau, e, yb, tb, yvpart));
      nl += 2;
    }
    const int kn = k0 + nb, m = n - kn;  // the trailing matrix
    FGLS_CUDA_TRY(launch_chained(tridiag_col_kernel, ceil_div(m, TR), 256, s, n, kn, nb, true, false, A, (long long)n,
                                 P, yb, tb, yvpart, nyv, tau, d, xb, npart));
    nl++;
    FGLS_CUDA_TRY(cudaGetLastError());
    // A -= [V W] [W V]^T; a short last panel leaves columns of P beyond nb unset
    double* T = A + kn + (long long)kn * n;
    if (nb == TB && dg && digit_gemm_pays(m, m, 2 * TB)) {
      DigitMulOpts lower;
      lower.c_lower = true;
      FGLS_CUDA_TRY(digit_dgemm(dg, s, false, true, m, m, 2 * TB, -1.0, P + kn, n, P + kn + (long long)TB * n, n, 1.0, T,
                                n, lower));
      symmetrize_kernel<<<dim3(ceil_div(m, 32), ceil_div(m, 32)), 256, 0, s>>>(m, T, n, T, n, nullptr);
      nl++;
    } else if (nb == TB) {
      FGLS_CUDA_TRY(dgemm(s, false, true, m, m, 2 * TB, -1.0, P + kn, n, P + kn + (long long)TB * n, n, 1.0, T, n));
    } else {
      FGLS_CUDA_TRY(dgemm(s, false, true, m, m, nb, -1.0, P + kn, n, P + kn + (long long)TB * n, n, 1.0, T, n));
      FGLS_CUDA_TRY(dgemm(s, false, true, m, m, nb, -1.0, P + kn + (long long)TB * n, n, P + kn, n, 1.0, T, n));
    }
  }
  tridiag_tail_kernel<<<1, 1, 0, s>>>(n, A, n, d, e);
  nl++;
  FGLS_CUDA_TRY(cudaGetLastError());
  mark(1);
  mark(2);  // (no explicit Q: the reflectors are applied to the eigenvectors below)
  // 3. eigenpairs of T by divide and conquer (fgls_dc.cu) into Z; A keeps the reflectors
  // one workspace for the divide and conquer, then for the back-transform
  // (Y: n x NBT, G, T: NBT x NBT, W, W2: NBT x n)
  constexpr int NBT = 512;  // K of the widest product; the back-transform at n = 5000: 35 ms with 256, 18 with 512
  const size_t bt_bytes = sizeof(double) * ((size_t)3 * NBT * n + (size_t)2 * NBT * NBT);
  void* dcw = nullptr;
  const size_t dcb = std::max(dc_workspace_bytes(n), bt_bytes);
  cudaError_t room = cudaMalloc(&dcw, dcb);
  if (room == cudaErrorMemoryAllocation && digit_gemm_trim(dg)) {  // FP64 products from here, in the digits' place
    (void)cudaGetLastError();
    dg = nullptr;
    room = cudaMalloc(&dcw, dcb);
  }
  FGLS_CUDA_TRY(room);
  FGLS_CUDA_TRY(cudaMemsetAsync(dfail, 0, sizeof(int), s));
  cudaError_t rc = dc_tridiag_eig(s, dg, n, d, e, W, Z, dcw, dfail, &nl);
  unscale_kernel<<<ceil_div(n, 256), 256, 0, s>>>(n, W, top);
  nl++;
  mark(3);
  // 4. Z := H_0 H_1 ... H_{n-3} Z, blocks of NB reflectors from the last one
  //    in compact-WY form (I - Y T Y^T): three FP64 products per block, 2 n^3
  //    flops in all -- what one with an explicit Q costs, without forming Q.
  {
    constexpr int NB = NBT;  // wide blocks: the Y^T Z product has NB/64 x n/64 output tiles
    double* Yb = (double*)dcw;         // n x NB
    double* G = Yb + (size_t)n * NB;   // NB x NB
    double* Tm = G + (size_t)NB * NB;  // NB x NB
    double* Wb = Tm + (size_t)NB * NB; // NB x n
    double* W2 = Wb + (size_t)NB * n;  // NB x n
    const int nref = n - 2;            // reflectors 0 .. n-3
    for (int b = nref > 0 ? ((nref - 1) / NB) * NB : -1; b >= 0 && rc == cudaSuccess; b -= NB) {
      const int nb = std::min(NB, nref - b);
      const int mr = n - b - 1;
      double* Zs = Z + (b + 1);  // rows b+1 .. n-1, all n columns (ld n)
      build_y_kernel<<<grid_for((long long)mr * nb), 256, 0, s>>>(n, b, nb, A, n, Yb);
      // G = Y^T Y has few output tiles: K split over the SMs either way (W2 as scratch)
      if (dg && digit_gemm_pays(nb, nb, mr))
        rc = digit_dgemm(dg, s, true, false, nb, nb, mr, 1.0, Yb, mr, Yb, mr, 0.0, G, nb);
      else
        rc = dgemm_splitk(s, true, false, nb, nb, mr, 1.0, Yb, mr, Yb, mr, 0.0, G, nb, W2, (long long)NB * n);
      if (rc == cudaSuccess) rc = larft(s, nb, tau + b, G, Tm, W2, &nl);
      if (rc == cudaSuccess) rc = digit_dgemm(dg, s, true, false, nb, n, mr, 1.0, Yb, mr, Zs, n, 0.0, Wb, nb);
      if (rc == cudaSuccess) rc = digit_dgemm(dg, s, false, false, nb, n, nb, 1.0, Tm, nb, Wb, nb, 0.0, W2, nb);
      if (rc == cudaSuccess) rc = digit_dgemm(dg, s, false, false, mr, n, nb, -1.0, Yb, mr, W2, nb, 1.0, Zs, n);
      nl++;
    }
  }
  int hfail = 0;
  if (rc == cudaSuccess) rc = cudaMemcpyAsync(&hfail, dfail, sizeof(int), cudaMemcpyDeviceToHost, s);
  if (rc == cudaSuccess) rc = cudaStreamSynchronize(s);
  cudaFree(dcw);
  digit_gemm_trim(dg);
  FGLS_CUDA_TRY(rc);
  *fail_out = hfail;
  mark(4);
  if (timing) {
    cudaEventSynchronize(ev[4]);
    float t[4];
    for (int i = 0; i < 4; i++) cudaEventElapsedTime(&t[i], ev[i], ev[i + 1]);
    fprintf(stderr, "[fgls eig n=%d] tridiagonal %.1f ms, divide-and-conquer %.1f ms, back-transform %.1f ms\n", n,
            t[0], t[2], t[3]);
    for (auto& x : ev) cudaEventDestroy(x);
  }
  if (launches) *launches += nl;
  note_launch(nl);
  return cudaSuccess;
}

}  // namespace fgls
