// Null-model REML fit of the variance components (h_j, sigma_j) per trait,
// FP64, in the eigenbasis of Phi (Phi = Z diag(w) Z^T).
//
// The reference takes h and sigma as inputs (src/fgls_chol.c:139-145 reads
// h2_path and sigma2_path; src/fgls_chol.c:251-256 and src/fgls_eigen.c:1085-1160
// use them as M_j = sigma_j (h_j Phi + (1 - h_j) I)).  This kernel estimates
// them from the same eigenbasis operands the association uses
// (ZtXL = Z^T XL, ZtY = Z^T Y, w).
//
// With d_l = 1/(1 + h (w_l - 1)) (sigma = 1):
//   G = sum_l d_l x_l x_l^T,  g = sum_l d_l x_l ytil_l,  b = G^-1 g,
//   r = ytil - ZtXL b,        q = sum_l d_l r_l^2.
// sigma is profiled out in closed form, sigma_hat(h) = q / (n - wXL), and the
// profiled REML log-likelihood (constants dropped) is
//   l_p(h)  = -1/2 [ (n-wXL) log sigma_hat - sum_l log d_l + log det G + (n-wXL) ],
//   l_p'(h) = -1/2 [ (n-wXL) q_c / q - sum_l c_l / d_l + tr(G^-1 G_c) ],
// c_l = dd_l/dh = -(w_l - 1) d_l^2, G_c = sum c x x^T, q_c = sum c r^2 (the
// b-derivative of q vanishes because b minimises q).  At sigma = sigma_hat(h)
// these are the REML value and h-gradient of the adjoint's null model.
//
// Maximisation over [lo, hi] follows EMMA (Kang et al., Genetics 178:1709,
// 2008): l_p and l_p' on an even grid, every + -> - sign change of l_p'
// refined to a root by bracketed secant steps, an
// endpoint taken when l_p' points out of the interval there, and the candidate
// with the largest l_p kept.
//
// Bound by FP64 issue (an SM takes a warp's FP64 instruction in 16 cycles), so
// every evaluation is kept short:
//   reml_common   what a grid point needs that no trait changes (d, c, the factor of
//                 G, log det G, tr G^-1 G_c and the sums of log d and c/d): once per
//                 grid point instead of once per grid point and trait
//   reml_grid     g, b and the residual sums of four traits at a grid point: 3 + 2 WX
//                 operations an element, against about 100 for a whole evaluation
//   reml_refine   a CTA per trait: the brackets' roots from evaluations of the
//                 gradient alone (no logarithms, reciprocals on a short chain), and
//                 one whole evaluation at each root
// n = 4001, 4 covariates, 100 traits: 13.9 -> 1.2 ms.  All sums have a fixed order.
#include <algorithm>
#include <cmath>

#include "fgls_common.cuh"
#include "fgls_kernels.cuh"

namespace fgls {

namespace {

constexpr int RF_THREADS = 256;
constexpr int RF_WARPS = RF_THREADS / 32;
constexpr int FGLS_REML_MAX_ITER = 100;  // steps per bracket

// Block-wide sums of K per-thread values, fixed order (warp butterfly, then
// warps in index order).  out[] is shared; all threads return after it is set.
template <int K>
__device__ __forceinline__ void block_sums(double (&v)[K], double* red, double* out) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < K; k++) {
    double x = v[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane == 0) red[w * K + k] = x;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < K; k += RF_THREADS) {
    double s = 0.0;
    for (int q = 0; q < RF_WARPS; q++) s += red[q * K + k];
    out[k] = s;
  }
  __syncthreads();
}

struct RemlPoint {
  double ll, dll, sig;
  int ok;
};

template <int WX>
struct RemlShared {
  static constexpr int NG = WX * (WX + 1) / 2;
  static constexpr int K1 = 2 * NG + WX + 3;  // G, G_c, g, sum log d, sum c/d, bad count
  double red[RF_WARPS * K1];
  double sums[K1];
  double b[WX];
  double logdet, tr, sl, sc;
  int ok;
  RemlPoint pt;
};

// l_p, l_p' and sigma_hat at h for the trait whose columns are X (n x WX,
// ld n) and y.  Called by all threads; the result is in S.pt.
template <int WX>
__device__ void reml_point(int n, double h, const double* __restrict__ W, const double* __restrict__ X,
                           const double* __restrict__ y, RemlShared<WX>& S) {
  constexpr int NG = RemlShared<WX>::NG, K1 = RemlShared<WX>::K1;
  double acc[K1];
#pragma unroll
  for (int k = 0; k < K1; k++) acc[k] = 0.0;
  for (int l = threadIdx.x; l < n; l += RF_THREADS) {
    const double wm = W[l] - 1.0;
    const double den = fma(h, wm, 1.0);
    const double d = 1.0 / den;
    const double c = -wm * d * d;
    double x[WX];
#pragma unroll
    for (int a = 0; a < WX; a++) x[a] = X[l + (long long)a * n];
    const double yl = y[l];
    int k = 0;
#pragma unroll
    for (int a = 0; a < WX; a++)
#pragma unroll
      for (int b = 0; b <= a; b++, k++) {
        const double xx = x[a] * x[b];
        acc[k] = fma(d, xx, acc[k]);
        acc[NG + k] = fma(c, xx, acc[NG + k]);
      }
#pragma unroll
    for (int a = 0; a < WX; a++) acc[2 * NG + a] = fma(d * x[a], yl, acc[2 * NG + a]);
    acc[2 * NG + WX] -= log(den);      // log d
    acc[2 * NG + WX + 1] -= wm * d;    // c / d
    acc[2 * NG + WX + 2] += (den > 0.0 && den < INFINITY) ? 0.0 : 1.0;
  }
  block_sums<K1>(acc, S.red, S.sums);
  if (threadIdx.x == 0) {
    double G[WX * WX], L[WX * WX];
    int k = 0;
    for (int a = 0; a < WX; a++)
      for (int b = 0; b <= a; b++, k++) {
        G[a + b * WX] = G[b + a * WX] = S.sums[NG + k];  // G_c
        L[a + b * WX] = L[b + a * WX] = S.sums[k];       // G
      }
    bool ok = S.sums[2 * NG + WX + 2] == 0.0;
    // Cholesky of G in place (lower)
    for (int j = 0; ok && j < WX; j++) {
      double v = L[j + j * WX];
      for (int q = 0; q < j; q++) v -= L[j + q * WX] * L[j + q * WX];
      if (!(v > 0.0)) {
        ok = false;
        break;
      }
      const double ljj = sqrt(v);
      L[j + j * WX] = ljj;
      for (int i = j + 1; i < WX; i++) {
        double u = L[i + j * WX];
        for (int q = 0; q < j; q++) u -= L[i + q * WX] * L[j + q * WX];
        L[i + j * WX] = u / ljj;
      }
    }
    double logdet = 0.0, tr = 0.0;
    if (ok) {
      double bb[WX];
      for (int a = 0; a < WX; a++) {
        logdet += 2.0 * log(L[a + a * WX]);
        bb[a] = S.sums[2 * NG + a];
      }
      // b = G^-1 g, and tr(G^-1 G_c) column by column
      for (int col = -1; col < WX; col++) {
        double v[WX];
        for (int a = 0; a < WX; a++) v[a] = col < 0 ? bb[a] : G[a + col * WX];
        for (int i = 0; i < WX; i++) {
          double u = v[i];
          for (int q = 0; q < i; q++) u -= L[i + q * WX] * v[q];
          v[i] = u / L[i + i * WX];
        }
        for (int i = WX - 1; i >= 0; i--) {
          double u = v[i];
          for (int q = i + 1; q < WX; q++) u -= L[q + i * WX] * v[q];
          v[i] = u / L[i + i * WX];
        }
        if (col < 0)
          for (int a = 0; a < WX; a++) S.b[a] = v[a];
        else
          tr += v[col];
      }
    }
    S.logdet = logdet;
    S.tr = tr;
    S.sl = S.sums[2 * NG + WX];
    S.sc = S.sums[2 * NG + WX + 1];
    S.ok = ok;
  }
  __syncthreads();
  double acc2[2] = {0.0, 0.0};
  if (S.ok) {
    double bl[WX];
#pragma unroll
    for (int a = 0; a < WX; a++) bl[a] = S.b[a];
    for (int l = threadIdx.x; l < n; l += RF_THREADS) {
      const double wm = W[l] - 1.0;
      const double d = 1.0 / fma(h, wm, 1.0);
      double r = y[l];
#pragma unroll
      for (int a = 0; a < WX; a++) r = fma(-X[l + (long long)a * n], bl[a], r);
      const double dr2 = d * r * r;
      acc2[0] += dr2;
      acc2[1] = fma(-wm * d, dr2, acc2[1]);  // c r^2 = -(w - 1) d * d r^2
    }
  }
  block_sums<2>(acc2, S.red, S.sums);  // pass-1 sums are consumed by now
  if (threadIdx.x == 0) {
    const double nn = (double)(n - WX);
    const double q = S.sums[0], qc = S.sums[1];
    RemlPoint p;
    p.ok = S.ok && q > 0.0 && isfinite(q);
    p.sig = p.ok ? q / nn : NAN;
    p.ll = p.ok ? -0.5 * (nn * log(p.sig) - S.sl + S.logdet + nn) : -INFINITY;
    p.dll = p.ok ? -0.5 * (nn * qc / q - S.sc + S.tr) : NAN;
    S.pt = p;
  }
  __syncthreads();
}

// Sums over a warp of K values a lane; value k's sum ends in v[0] of lane k (K <=
// 32) or of lanes k, with v[1] for value 32 + k (K <= 64).  Each round halves the
// values a lane carries: K additions instead of 5 K.
template <int K>
__device__ __forceinline__ void warp_sums(double (&v)[K]) {
  const int lane = threadIdx.x & 31;
  static_assert(K == 32 || K == 64, "padded");
#pragma unroll
  for (int u = 0; u < K / 32; u++) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const bool up = lane & o;
#pragma unroll
      for (int k = 0; k < o; k++) {
        const double send = up ? v[32 * u + k] : v[32 * u + k + o], keep = up ? v[32 * u + k + o] : v[32 * u + k];
        v[32 * u + k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
  }
#pragma unroll
  for (int u = 1; u < K / 32; u++) v[u] = v[32 * u];
}

// One warp: from the sums of G (packed lower), G_c and g, the factor L of G
// (reciprocal diagonal in rd), log det G, tr G^-1 G_c and b = G^-1 g.  Lane c < WX
// solves for column c of G_c, lane WX for g; every lane returns the same values.
template <int WX>
__device__ __forceinline__ bool warp_model(const double* __restrict__ G, const double* __restrict__ Gc,
                                           const double* __restrict__ g, double (&L)[WX][WX], double (&rd)[WX],
                                           double& tr, double (&b)[WX]) {
  const int lane = threadIdx.x & 31;
  bool ok = true;
#pragma unroll
  for (int j = 0; j < WX; j++) {
    double v = G[j * (j + 1) / 2 + j];
#pragma unroll
    for (int q = 0; q < j; q++) v = fma(-L[j][q], L[j][q], v);
    ok = ok && v > 0.0;
    rd[j] = rsqrt(v);
    L[j][j] = v * rd[j];
#pragma unroll
    for (int i = j + 1; i < WX; i++) {
      double u = G[i * (i + 1) / 2 + j];
#pragma unroll
      for (int q = 0; q < j; q++) u = fma(-L[i][q], L[j][q], u);
      L[i][j] = u * rd[j];
    }
  }
  double v[WX];
#pragma unroll
  for (int a = 0; a < WX; a++) {
    const int hi = max(a, lane), lo = min(a, lane);
    v[a] = lane < WX ? Gc[hi * (hi + 1) / 2 + lo] : g ? g[a] : 0.0;
  }
#pragma unroll
  for (int i = 0; i < WX; i++) {
#pragma unroll
    for (int q = 0; q < i; q++) v[i] = fma(-L[i][q], v[q], v[i]);
    v[i] *= rd[i];
  }
#pragma unroll
  for (int i = WX - 1; i >= 0; i--) {
#pragma unroll
    for (int q = i + 1; q < WX; q++) v[i] = fma(-L[q][i], v[q], v[i]);
    v[i] *= rd[i];
  }
  tr = 0.0;
#pragma unroll
  for (int a = 0; a < WX; a++) {
    tr += __shfl_sync(0xffffffffu, v[a], a);
    b[a] = __shfl_sync(0xffffffffu, v[a], WX);
  }
  return ok;
}

template <int WX>
struct RemlCommon {  // of a grid point
  double L[WX][WX], rd[WX], logdet, tr, sl, sc;
  int ok;
};

__device__ __forceinline__ double grid_h(int k, int grid, double lo, double hi) {
  return k == grid - 1 ? hi : lo + (hi - lo) * ((double)k / (grid - 1));
}

template <int WX>
__global__ void __launch_bounds__(RF_THREADS)
    reml_common_kernel(int n, const double* __restrict__ W, const double* __restrict__ X, double lo, double hi, int grid,
                       int k0, double* __restrict__ dtab, RemlCommon<WX>* __restrict__ common) {
  constexpr int NG = WX * (WX + 1) / 2, K1 = 2 * NG + 2, KP = K1 <= 32 ? 32 : 64;
  __shared__ double red[RF_WARPS][64], sums[64];
  __shared__ int sbad;
  const double h = grid_h(k0 + blockIdx.x, grid, lo, hi);
  double* dt = dtab + (long long)blockIdx.x * 2 * n;
  double acc[KP];
#pragma unroll
  for (int k = 0; k < KP; k++) acc[k] = 0.0;
  int bad = 0;
  if (threadIdx.x == 0) sbad = 0;
  __syncthreads();
  for (int l = threadIdx.x; l < n; l += RF_THREADS) {
    const double wm = W[l] - 1.0;
    const double den = fma(h, wm, 1.0);
    const int hb = __double2hiint(den);
    bad |= !(den > 0.0) || hb >= 0x7ff00000;
    const double d = 1.0 / den;
    const double c = -wm * d * d;
    dt[l] = d;
    dt[n + l] = c;
    double x[WX];
#pragma unroll
    for (int a = 0; a < WX; a++) x[a] = X[l + (long long)a * n];
    int k = 0;
#pragma unroll
    for (int a = 0; a < WX; a++)
#pragma unroll
      for (int b = 0; b <= a; b++, k++) {
        const double xx = x[a] * x[b];
        acc[k] = fma(d, xx, acc[k]);
        acc[NG + k] = fma(c, xx, acc[NG + k]);
      }
    acc[2 * NG] -= log(den);   // log d
    acc[2 * NG + 1] -= wm * d;  // c / d
  }
  if (bad) sbad = 1;
  warp_sums<KP>(acc);
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  red[wp][lane] = acc[0];
  if (KP > 32) red[wp][32 + lane] = acc[1];
  __syncthreads();
  if (threadIdx.x < KP) {
    double s = 0.0;
    for (int q = 0; q < RF_WARPS; q++) s += red[q][threadIdx.x];
    sums[threadIdx.x] = s;
  }
  __syncthreads();
  if (wp == 0) {
    RemlCommon<WX> r;
    double b[WX];
    const bool ok = warp_model<WX>(sums, sums + NG, nullptr, r.L, r.rd, r.tr, b);
    r.logdet = 0.0;
#pragma unroll
    for (int a = 0; a < WX; a++) r.logdet += 2.0 * log(r.L[a][a]);
    r.sl = sums[2 * NG];
    r.sc = sums[2 * NG + 1];
    r.ok = ok && !sbad;
    if (lane == 0) common[blockIdx.x] = r;
  }
}

// Four traits at a grid point: out[(j*grid + k)*3 ..] = ll, dll, sigma.
constexpr int GT_THREADS = 128, GT_TRAITS = 4;
template <int WX>
__global__ void __launch_bounds__(GT_THREADS)
    reml_grid_kernel(int n, int t, const double* __restrict__ X, const double* __restrict__ Y, int grid, int k0,
                     const double* __restrict__ dtab, const RemlCommon<WX>* __restrict__ common,
                     double* __restrict__ out) {
  __shared__ double red[GT_THREADS / 32][32], bs[GT_TRAITS][WX];
  const RemlCommon<WX>& cm = common[blockIdx.x];
  const double* dt = dtab + (long long)blockIdx.x * 2 * n;
  const int j0 = blockIdx.y * GT_TRAITS, nt = min(GT_TRAITS, t - j0);
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const double* y[GT_TRAITS];
#pragma unroll
  for (int u = 0; u < GT_TRAITS; u++) y[u] = Y + (long long)(j0 + min(u, nt - 1)) * n;
  double acc[32];
#pragma unroll
  for (int k = 0; k < 32; k++) acc[k] = 0.0;
  for (int l = threadIdx.x; l < n; l += GT_THREADS) {
    const double d = dt[l];
    double x[WX];
#pragma unroll
    for (int a = 0; a < WX; a++) x[a] = X[l + (long long)a * n];
#pragma unroll
    for (int u = 0; u < GT_TRAITS; u++) {
      const double dy = d * y[u][l];
#pragma unroll
      for (int a = 0; a < WX; a++) acc[u * WX + a] = fma(x[a], dy, acc[u * WX + a]);
    }
  }
  warp_sums<32>(acc);
  red[wp][lane] = acc[0];
  __syncthreads();
  if (threadIdx.x < GT_TRAITS) {  // b = G^-1 g of a trait per thread
    double v[WX];
#pragma unroll
    for (int a = 0; a < WX; a++) {
      v[a] = 0.0;
      for (int q = 0; q < GT_THREADS / 32; q++) v[a] += red[q][threadIdx.x * WX + a];
    }
#pragma unroll
    for (int i = 0; i < WX; i++) {
#pragma unroll
      for (int q = 0; q < i; q++) v[i] = fma(-cm.L[i][q], v[q], v[i]);
      v[i] *= cm.rd[i];
    }
#pragma unroll
    for (int i = WX - 1; i >= 0; i--) {
#pragma unroll
      for (int q = i + 1; q < WX; q++) v[i] = fma(-cm.L[q][i], v[q], v[i]);
      v[i] *= cm.rd[i];
    }
#pragma unroll
    for (int a = 0; a < WX; a++) bs[threadIdx.x][a] = v[a];
  }
  __syncthreads();
  double b[GT_TRAITS][WX], rs[2 * GT_TRAITS];
#pragma unroll
  for (int u = 0; u < GT_TRAITS; u++) {
    rs[2 * u] = rs[2 * u + 1] = 0.0;
#pragma unroll
    for (int a = 0; a < WX; a++) b[u][a] = bs[u][a];
  }
  for (int l = threadIdx.x; l < n; l += GT_THREADS) {
    const double d = dt[l], c = dt[n + l];
    double x[WX];
#pragma unroll
    for (int a = 0; a < WX; a++) x[a] = X[l + (long long)a * n];
#pragma unroll
    for (int u = 0; u < GT_TRAITS; u++) {
      double r = y[u][l];
#pragma unroll
      for (int a = 0; a < WX; a++) r = fma(-x[a], b[u][a], r);
      const double r2 = r * r;
      rs[2 * u] = fma(d, r2, rs[2 * u]);
      rs[2 * u + 1] = fma(c, r2, rs[2 * u + 1]);
    }
  }
#pragma unroll
  for (int k = 0; k < 32; k++) acc[k] = k < 2 * GT_TRAITS ? rs[k] : 0.0;
  warp_sums<32>(acc);
  __syncthreads();
  red[wp][lane] = acc[0];
  __syncthreads();
  if ((int)threadIdx.x < nt) {
    double q = 0.0, qc = 0.0;
    for (int w = 0; w < GT_THREADS / 32; w++) {
      q += red[w][2 * threadIdx.x];
      qc += red[w][2 * threadIdx.x + 1];
    }
    const double nn = (double)(n - WX);
    const bool ok = cm.ok && q > 0.0 && isfinite(q);
    const double sig = ok ? q / nn : NAN;
    double* o = out + ((long long)(j0 + threadIdx.x) * grid + k0 + blockIdx.x) * 3;
    o[0] = ok ? -0.5 * (nn * log(sig) - cm.sl + cm.logdet + nn) : -INFINITY;
    o[1] = ok ? -0.5 * (nn * qc / q - cm.sc + cm.tr) : NAN;
    o[2] = sig;
  }
}

template <int WX>
struct GradShared {
  double red[RF_WARPS][64], sums[64], b[WX], tr;
  int ok, bad;
};
// l_p' at h and the size of its terms; *ok false where the model is not positive
// definite there.  All threads of the CTA call it and get the result.
template <int WX>
__device__ double reml_gradient(int n, double h, const double* __restrict__ W, const double* __restrict__ X,
                                const double* __restrict__ y, GradShared<WX>& S, bool* ok, double* size) {
  constexpr int NG = WX * (WX + 1) / 2, K1 = 2 * NG + WX + 1, KP = K1 <= 32 ? 32 : 64;
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  double acc[KP];
#pragma unroll
  for (int k = 0; k < KP; k++) acc[k] = 0.0;
  int bad = 0;
  __syncthreads();
  if (threadIdx.x == 0) S.bad = 0;
  __syncthreads();
  for (int l = threadIdx.x; l < n; l += RF_THREADS) {
    const double wm = W[l] - 1.0;
    const double den = fma(h, wm, 1.0);
    bad |= !(__double2hiint(den) > 0) || __double2hiint(den) >= 0x7ff00000;
    const double d = chain_rcp(den);
    const double wd = wm * d, c = -wd * d;
    double x[WX];
#pragma unroll
    for (int a = 0; a < WX; a++) x[a] = X[l + (long long)a * n];
    const double dy = d * y[l];
    int k = 0;
#pragma unroll
    for (int a = 0; a < WX; a++) {
      acc[2 * NG + a] = fma(x[a], dy, acc[2 * NG + a]);
#pragma unroll
      for (int b = 0; b <= a; b++, k++) {
        const double xx = x[a] * x[b];
        acc[k] = fma(d, xx, acc[k]);
        acc[NG + k] = fma(c, xx, acc[NG + k]);
      }
    }
    acc[2 * NG + WX] -= wd;  // c / d
  }
  if (bad) S.bad = 1;
  warp_sums<KP>(acc);
  S.red[wp][lane] = acc[0];
  if (KP > 32) S.red[wp][32 + lane] = acc[1];
  __syncthreads();
  if (threadIdx.x < KP) {
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < RF_WARPS; q++) s += S.red[q][threadIdx.x];
    S.sums[threadIdx.x] = s;
  }
  __syncthreads();
  if (wp == 0) {
    double L[WX][WX], rd[WX], tr, b[WX];
    const bool good = warp_model<WX>(S.sums, S.sums + NG, S.sums + 2 * NG, L, rd, tr, b);
    if (lane == 0) {
      S.ok = good && !S.bad;
      S.tr = tr;
#pragma unroll
      for (int a = 0; a < WX; a++) S.b[a] = b[a];
    }
  }
  __syncthreads();
  double bl[WX], q = 0.0, qc = 0.0;
#pragma unroll
  for (int a = 0; a < WX; a++) bl[a] = S.b[a];
  for (int l = threadIdx.x; l < n; l += RF_THREADS) {
    const double wm = W[l] - 1.0;
    const double d = chain_rcp(fma(h, wm, 1.0));
    double r = y[l];
#pragma unroll
    for (int a = 0; a < WX; a++) r = fma(-X[l + (long long)a * n], bl[a], r);
    const double dr2 = d * r * r;
    q += dr2;
    qc = fma(-wm * d, dr2, qc);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    q += __shfl_xor_sync(0xffffffffu, q, o);
    qc += __shfl_xor_sync(0xffffffffu, qc, o);
  }
  if (lane == 0) {
    S.red[wp][0] = q;
    S.red[wp][1] = qc;
  }
  __syncthreads();
  q = qc = 0.0;
#pragma unroll
  for (int u = 0; u < RF_WARPS; u++) {
    q += S.red[u][0];
    qc += S.red[u][1];
  }
  *ok = S.ok && q > 0.0 && isfinite(q);
  const double ratio = (double)(n - WX) * qc / q, sc = S.sums[2 * NG + WX];
  *size = fabs(ratio) + fabs(sc) + fabs(S.tr);
  return -0.5 * (ratio - sc + S.tr);
}

// One CTA per trait: the candidates' maximum from the grid's values (gp: ll, dll,
// sigma of each point).
template <int WX>
__global__ void __launch_bounds__(RF_THREADS)
    reml_refine_kernel(int n, int t, const double* __restrict__ W, const double* __restrict__ ZtXL,
                       const double* __restrict__ ZtY, double lo, double hi, int grid, const double* __restrict__ gp,
                       double* __restrict__ out, DevStatus* st) {
  __shared__ RemlShared<WX> S;
  __shared__ GradShared<WX> D;
  __shared__ double g[FGLS_REML_MAX_GRID * 3];
  __shared__ int sok;
  const int j = blockIdx.x;
  const double* y = ZtY + (long long)j * n;
  if (threadIdx.x == 0) sok = 1;
  __syncthreads();
  for (int k = threadIdx.x; k < 3 * grid; k += RF_THREADS) {
    g[k] = gp[(long long)j * grid * 3 + k];
    if (k % 3 == 1 && isnan(g[k])) sok = 0;
  }
  __syncthreads();
  auto hk = [&](int k) { return grid_h(k, grid, lo, hi); };
  auto gll = [&](int k) { return g[3 * k]; };
  auto gdll = [&](int k) { return g[3 * k + 1]; };
  auto gsig = [&](int k) { return g[3 * k + 2]; };
  bool ok = sok;
  double bh = NAN, bll = -INFINITY, bsig = NAN, bdll = NAN;
  if (ok) {
    if (!(gdll(0) > 0.0)) bh = lo, bll = gll(0), bsig = gsig(0), bdll = gdll(0);
    if (gdll(grid - 1) >= 0.0 && gll(grid - 1) > bll)
      bh = hi, bll = gll(grid - 1), bsig = gsig(grid - 1), bdll = gdll(grid - 1);
    for (int k = 0; k + 1 < grid && ok; k++) {
      if (!(gdll(k) > 0.0 && !(gdll(k + 1) > 0.0))) continue;
      // root of l_p' in [a, b], l_p'(a) > 0 >= l_p'(b): secant steps, bisection
      // where one leaves the bracket or they have not ended after a dozen.  Ends with
      // the bracket or a step below the tolerance, or with a gradient below half an
      // ulp of its own terms, whose sign is nothing but rounding: four evaluations a
      // root, where the Illinois rule, ending by the bracket alone, took 8 and on
      // some traits 35 (the launch lasts as long as its slowest trait).
      double a = hk(k), b = hk(k + 1), x0 = a, f0 = gdll(k), x = b, fx = gdll(k + 1);
      if (fabs(f0) < fabs(fx)) {
        x0 = b, f0 = fx;
        x = a, fx = gdll(k);
      }
      for (int it = 0; it < FGLS_REML_MAX_ITER && fx != 0.0; it++) {
        double xn = fx != f0 ? x - fx * (x - x0) / (fx - f0) : a;
        if (!(xn > a && xn < b) || (it >= 12 && (it & 1))) xn = 0.5 * (a + b);
        const double tol = 1e-15 + 2e-16 * fabs(xn);
        const bool last = fabs(xn - x) <= tol;
        x0 = x, f0 = fx;
        x = xn;
        if (last) break;
        double size;
        fx = reml_gradient<WX>(n, x, W, ZtXL, y, D, &ok, &size);
        if (!ok || fabs(fx) <= 1.1e-16 * size) break;
        if (fx > 0.0) a = x;
        else b = x;
        if (b - a <= tol) break;
      }
      if (!ok) break;
      __syncthreads();
      reml_point<WX>(n, x, W, ZtXL, y, S);
      ok = S.pt.ok;
      if (ok && S.pt.ll > bll) bh = x, bll = S.pt.ll, bsig = S.pt.sig, bdll = S.pt.dll;
      __syncthreads();
    }
  }
  if (threadIdx.x == 0) {
    if (!ok || !(bll > -INFINITY)) {
      bh = bsig = bll = bdll = NAN;
      set_status(st, FGLSGPU_ENOTSPD, -2, j);
    }
    out[j] = bh;
    out[t + j] = bsig;
    out[2 * t + j] = bll;
    out[3 * t + j] = bdll;
  }
}

// grid points a pass: their d and c within 256 MB
int grid_chunk(int n, int grid) { return (int)std::max<long long>(1, std::min<long long>(grid, (16LL << 20) / n)); }

template <int WX>
void launch_reml(cudaStream_t s, int n, int t, const double* W, const double* X, const double* Y, double lo, double hi,
                 int grid, double* work, double* out, DevStatus* st) {
  const int chunk = grid_chunk(n, grid);
  double* gp = work;                               // t x grid x 3
  double* dtab = gp + (size_t)3 * t * grid;        // chunk x 2 x n
  RemlCommon<WX>* cm = (RemlCommon<WX>*)(dtab + (size_t)2 * chunk * n);
  for (int k0 = 0; k0 < grid; k0 += chunk) {
    const int kc = std::min(chunk, grid - k0);
    reml_common_kernel<WX><<<kc, RF_THREADS, 0, s>>>(n, W, X, lo, hi, grid, k0, dtab, cm);
    reml_grid_kernel<WX><<<dim3(kc, ceil_div(t, GT_TRAITS)), GT_THREADS, 0, s>>>(n, t, X, Y, grid, k0, dtab, cm, gp);
    note_launch(2);
  }
  reml_refine_kernel<WX><<<t, RF_THREADS, 0, s>>>(n, t, W, X, Y, lo, hi, grid, gp, out, st);
  note_launch();
}

}  // namespace

size_t reml_workspace_bytes(int n, int t, int grid) {
  return sizeof(double) * ((size_t)3 * t * grid + (size_t)2 * grid_chunk(n, grid) * n) +
         (size_t)grid * sizeof(RemlCommon<FGLS_MAX_P - 1>) + 256;
}

cudaError_t reml_fit(cudaStream_t s, int n, int t, int wXL, const double* W, const double* ZtXL, const double* ZtY,
                     double lo, double hi, int grid, double* work, double* out, DevStatus* st) {
  if (t <= 0) return cudaSuccess;
  if (n <= wXL || grid < 2 || grid > FGLS_REML_MAX_GRID || !(lo >= 0.0 && lo < hi && hi <= 1.0))
    return cudaErrorInvalidValue;
  switch (wXL) {
#define FGLS_REML_CASE(WX) \
  case WX:                  \
    launch_reml<WX>(s, n, t, W, ZtXL, ZtY, lo, hi, grid, work, out, st); \
    break;
    FGLS_REML_CASE(1)
    FGLS_REML_CASE(2)
    FGLS_REML_CASE(3)
    FGLS_REML_CASE(4)
    FGLS_REML_CASE(5)
    FGLS_REML_CASE(6)
    FGLS_REML_CASE(7)
#undef FGLS_REML_CASE
    default:
      return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace fgls
