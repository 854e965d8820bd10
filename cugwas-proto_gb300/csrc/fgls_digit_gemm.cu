// FP64 matrix products as exact sums of FP8 digit products (tcgen05), the bulk
// arithmetic of the FP64 path and of the factorizations: GB300 runs FP64 FMAs
// at about 1.2 TFLOP/s and kind::f8f6f4 MMAs at 4.5 PFLOP/s.
//
//   C = alpha * A * B^T + beta * C,  A: M rows, B: N rows, K elements a row.
//
// Digits.  Row r of an operand is scaled by a power of two, 2^ex, so that
// |x| 2^-ex < 1/2, rounded to a multiple of 2^-60 and written in base 32 with
// signed digits, x 2^-ex = sum_{s=1..12} d_s 32^-s, |d_s| <= 16: exact in E4M3.
// The cut works on the bit pattern in integer instructions: the 60-bit fixed
// point magnitude plus sum_s 16 * 32^(12-s) has the digits d_s + 16 as its
// 5-bit fields.
//
// Products.  A product of digits s and t has weight 32^-(s+t); level L is the
// sum of all pairs with s + t = L.  Levels 2 .. 13 are kept (78 of the 144
// pairs); what is dropped is below 11 * 2^8 * 2^-70 = 2^-58.5 of the product of
// the row scales per element, and of random sign, like the rounding of the digits:
// for rows of one magnitude less than the rounding of an FP64 accumulation (what
// uses the products and holds mixed ones: the engine's diag_range_kernel).  Measured
// 2-norm errors over
// 150 entries against exactly rounded sums, normal data, digits / FP64 kernel:
// K = 128 5e-15 / 5e-14, K = 1000 3e-14 / 4e-13, K = 10000 1.2e-13 / 4.1e-12
// (hard calls as one operand 1.8e-15).  A level's sum over K is an integer;
// in units of the accumulator at most pairs * K * 2^8, so 65536 pairs x K of a
// level are summed exactly in FP32 and then added to int32 sums.  At the end
// the levels are combined in 128-bit integers and rounded once to FP64: no
// FP64 instruction runs per element unless alpha or beta asks for one.
// Operands with fewer digits (hard-call genotypes have one) have fewer pairs:
// the digits in use per 256 rows are found while cutting.
//
// digit_gemm_kernel: persistent clusters of two CTAs, 256 x 256 tiles with
// tcgen05.mma.cta_group::2 (M = 256, N = 256, K = 32), each CTA holding 128
// rows of A and 128 of B.  Two levels run at once, L in TMEM columns 0-255 and
// L + 1 in 256-511.  For a K-block the digits of B ascend, t = 1, 2, ..: the
// A tile that level L + 1 needs at step t, digit L + 1 - t, is the one level L
// used at step t - 1, so each step (one A tile, one B tile, at the first a second A
// tile) feeds eight MMAs and the previous step's A tile is kept one step
// longer.  That is 28 bytes per clock and SM from L2, half of what one A and one
// B tile per four MMAs would take.
//   warp 0     TMA producer (each CTA its own 128 rows), a ring of fourteen tiles
//   warp 1     MMA issue (pair leader), TMEM allocation
//   warps 2-17 epilogue: q = 32 P_L + P_{L+1} as int32 into the CTA's own
//              planes (L2-resident, 4 bytes per element and level pair); once a
//              tile's last pass is stored its TMEM is released and the planes
//              are combined while the next tile's MMAs run.
// Every wait is bounded as in fgls_ozaki.cu.
//
// Bound by the FP8 pipe: 10000 x 4096 x 10000 takes 18.1 ms with both cuts (78
// pairs: 3.5 PFLOP/s, 0.92 of twice the measured BF16 rate) and 3.7 ms with
// hard calls (12 pairs), where the FP64 kernel takes 665 ms.
#include <cuda.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <cmath>

#include "fgls_common.cuh"
#include "fgls_digit_gemm.cuh"
#include "fgls_kernels.cuh"
#include "fgls_tc.cuh"

namespace fgls {

namespace {

using namespace oz;

constexpr int ND = DG_DIGITS;
constexpr int ROW = 128;               // bytes (digits) of a K-step
constexpr int TILE = 128 * ROW;        // 16 KB: 128 rows of one digit plane
// Ring of tiles; a step takes two or three of them (an A tile, at a K-block's first
// step the A tile level L + 1 starts with, a B tile) and one of the barriers.  In
// fixed stages of three tiles four fit, in stages of two six, with a stage to
// itself for the third: 10000 x 4096 x 10000 took 19.1 and 18.6 ms, with hard calls
// (three tiles every step) 3.67 and 4.37; tile by tile 18.7 and 3.72.
constexpr int TILES = 14;
constexpr int STEPS = 8;               // at most TILES / 2 in flight
constexpr int SMEM = TILES * TILE + 1024 + 256;
constexpr int EPI_WARPS = 16;
constexpr int EPI_COLS = 256 * 4 / EPI_WARPS;  // columns of an epilogue warp (32 rows)
constexpr int NTHREADS = 64 + 32 * EPI_WARPS;
constexpr int MAXPASS = (ND + 1) / 2;  // level pairs
constexpr int PLANE4 = 128 * 256 / 4;   // int4s of one CTA's plane
constexpr int PAIR_K = 512;            // K-steps x pairs one FP32 accumulator takes exactly (65536 elements)
// int32 planes: 33 * 2^8 * pairs * K < 2^31 for 12 pairs
// tiles per cluster up to which the split form runs: with whole tiles as units the
// other clusters idle and a tile's six passes and its epilogue are one chain
// (301 x 74 x 301 with both cuts: 0.173 ms, split 0.080; 1000 x 512 x 64 0.144, 0.064)
constexpr double SPLIT_TILES = 1.0;
constexpr int K_MAX_STEPS = 160;       // 20480 elements of K per launch
// kind::f8f6f4: D=F32, A=B=E4M3, K-major, N=256, M=256 (the pair)
constexpr uint32_t DG_IDESC = (1u << 4) | ((uint32_t)(256 >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);

__device__ __forceinline__ void tma_load_3d_cg2(void* dst, const CUtensorMap* tm, int x, int y, int z, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, "
      "%4}], [%5];" ::"r"(smem_u32(dst)),
      "l"((uint64_t)tm), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}

struct DgArgs {
  int M, N;
  int kb0, nk;            // K-steps of this launch: [kb0, kb0 + nk)
  // Split form (few tiles): a unit is one level pair of a tile over a part of K;
  // level pair i is cut into zs[i] parts of kper[i] steps and every unit writes
  // its own plane.  zsum = 0: a unit is a whole tile.
  int zsum, zs[MAXPASS], kper[MAXPASS];
  int tiles_m, tiles_n;   // 256 x 256 tiles
  int lower_tiles;        // tiles are those with n_tile <= m_tile only, and only r >= c is written
  int a_lower;            // row r of A is zero beyond column r
  const int *exA, *exB, *ndA, *ndB;
  double alpha, beta;
  double* C;
  long long ldc;
  int4* planes;
  int* err;
  unsigned long long wait_ns;
};

// What the roles need of a unit: an output tile, level pairs [i0, i1) and a
// range of K; `slot`: the plane of a split unit.
struct Unit {
  int mt, nt, kb, nk, da, db, i0, i1, slot;
};
__device__ __forceinline__ int dg_tiles(const DgArgs& g) {
  return g.lower_tiles ? g.tiles_m * (g.tiles_m + 1) / 2 : g.tiles_m * g.tiles_n;
}
__device__ __forceinline__ int dg_units(const DgArgs& g) { return dg_tiles(g) * max(1, g.zsum); }
// Tile t.  Lower-triangular A: row tiles with the most K first (the units are
// dealt in order); else groups of eight row tiles, so that the tiles in flight
// share operand tiles in L2.
__device__ __forceinline__ void dg_tile(const DgArgs& g, int t, Unit& U) {
  if (g.lower_tiles) {
    int m = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
    while (m * (m + 1) / 2 > t) m--;
    while ((m + 1) * (m + 2) / 2 <= t) m++;
    U.mt = m;
    U.nt = t - m * (m + 1) / 2;
  } else if (g.a_lower) {
    U.mt = g.tiles_m - 1 - t / g.tiles_n;
    U.nt = t % g.tiles_n;
  } else {
    const int per = 8 * g.tiles_n, grp = t / per;
    const int gm = min(8, g.tiles_m - grp * 8);
    const int in = t - grp * per;
    U.mt = grp * 8 + in % gm;
    U.nt = in / gm;
  }
  U.da = max(1, g.ndA[U.mt]);
  U.db = max(1, g.ndB[U.nt]);
  U.i0 = 0;
  U.i1 = min(ND + 1, U.da + U.db) / 2;
  U.kb = g.kb0;
  U.nk = g.nk;
  if (g.a_lower) U.nk = min(U.nk, 2 * (U.mt + 1) - U.kb);  // 256 rows: 2 K-steps a row tile
  U.slot = 0;
}
// Unit u.  Split form: the level pairs with the most digit pairs first.
__device__ __forceinline__ Unit dg_unit(const DgArgs& g, int u) {
  Unit U;
  if (g.zsum == 0) {
    dg_tile(g, u, U);
    return U;
  }
  const int tiles = dg_tiles(g), t = u % tiles;
  int z = u / tiles, i = MAXPASS - 1;
  dg_tile(g, t, U);
  U.slot = t * g.zsum + z;
  while (z >= g.zs[i]) z -= g.zs[i--];
  U.i0 = i;
  U.i1 = min(i + 1, U.i1);
  U.kb += z * g.kper[i];
  U.nk = min(U.nk - z * g.kper[i], g.kper[i]);
  return U;
}

// Level pair i of a unit: levels L and L + 1, the B digits t that take part.
struct Pass {
  int L, tlo, thi, has1, pro, chunk;  // pro: step tlo brings A digit L + 1 - tlo too; chunk: K-steps a pass
};
__device__ __forceinline__ Pass dg_pass(const Unit& U, int i) {
  Pass P;
  const int lmax = min(ND + 1, U.da + U.db);
  P.L = 2 + 2 * i;
  P.has1 = P.L + 1 <= lmax;
  P.tlo = max(1, P.L - U.da);
  P.thi = P.has1 ? min(U.db, P.L) : min(U.db, P.L - 1);
  P.pro = P.has1 && P.L + 1 - P.tlo <= U.da;
  const int steps = max(1, U.nk), most = PAIR_K / (P.thi - P.tlo + 1);
  const int n = (steps + most - 1) / most;
  P.chunk = (steps + n - 1) / n;
  return P;
}

// An integer |v| <= 2^24 held in a float, as an int without a conversion
// instruction (those run at a quarter of the FP32 rate): the multiple of four
// by the 1.5 * 2^25 addend, the rest by the 1.5 * 2^23 one.
__device__ __forceinline__ int exact_f2i(float v) {
  const float t = __fadd_rn(v, 50331648.0f);
  const float r = __fsub_rn(v, __fsub_rn(t, 50331648.0f));
  const float u = __fadd_rn(r, 12582912.0f);
  return (int)(((uint32_t)__float_as_int(t) - 0x4C400000u) * 4u + ((uint32_t)__float_as_int(u) - 0x4B400000u));
}

constexpr int TOP = 0x7ff, ALL_PINF = 0x800, ALL_NINF = 0x1000, ALL_POS = 0x2000, ALL_NEG = 0x4000;  // below
// exponent of a row's scale from the largest biased exponent in it (what a
// DigitMat keeps per row)
__device__ __forceinline__ int row_exponent(int top) { return (top & TOP) - 1021; }
// What a DigitMat's ex holds of a row beside it: of a row with the exponent of NaN and
// infinities, whether all its non-finite elements are +inf or all -inf; of rows cut by
// digit_cut_signed, whether all elements are above or all below zero.
// The product of two rows of which one or both are not finite: infinite where the signs
// say so (what an FP64 sum gives), else NaN.
__device__ __forceinline__ double nonfinite_product(int a, int b) {
  const int inf = (a & TOP) == TOP ? a : b, fin = inf == a ? b : a;
  const bool known = (fin & TOP) != TOP && (inf & (ALL_PINF | ALL_NINF)) && (fin & (ALL_POS | ALL_NEG));
  const bool neg = ((inf & ALL_NINF) != 0) != ((fin & ALL_NEG) != 0);
  return __longlong_as_double(!known ? 0x7ff8000000000000ll : neg ? (long long)0xfff0000000000000ull : 0x7ff0000000000000ll);
}

// (W 2^sh + V) 2^e rounded to FP64 (to nearest even) in integer instructions;
// |W|, |V| < 2^52, sh <= 30.
__device__ __forceinline__ double combine_words(long long W, int sh, long long V, int e) {
  uint64_t lo = (uint64_t)W << sh;
  long long hi = sh ? W >> (64 - sh) : W >> 63;
  const uint64_t sum = lo + (uint64_t)V;
  hi += (V >> 63) + (sum < lo);
  lo = sum;
  const bool neg = hi < 0;
  if (neg) {
    lo = 0 - lo;
    hi = ~hi + (lo == 0);
  }
  // the magnitude (below 2^83) with its highest bit at bit 63 of m
  uint64_t m;
  int top;
  bool sticky = false;
  if (hi) {
    const int s = 32 - __clz((int)hi);  // 1 .. 19 bits above bit 63
    top = 63 + s;
    m = ((uint64_t)hi << (64 - s)) | (lo >> s);
    sticky = (lo << (64 - s)) != 0;
  } else {
    if (!lo) return 0.0;
    const int z = __clzll((long long)lo);
    top = 63 - z;
    m = lo << z;
  }
  const uint32_t rest = (uint32_t)m & 0x7ffu;
  m >>= 11;
  m += (rest > 0x400u || (rest == 0x400u && (sticky || (m & 1)))) ? 1 : 0;
  const int ex = top + e;  // m in [2^52, 2^53]
  if (ex < -1000 || ex > 1000) return ldexp(neg ? -(double)m : (double)m, ex - 52);
  return __longlong_as_double((long long)((m + ((uint64_t)(ex + 1022) << 52)) | (neg ? 1ull << 63 : 0ull)));
}

// Four elements of row r from column c on: T = sum_i q_i 2^(10 (np - 1 - i)),
// the element is T 2^(exA + exB - 5 (2 np + 1)); alpha, beta and the write.
__device__ __forceinline__ void store_four(const DgArgs& g, const int4 (&q)[MAXPASS], int np, int r, int c) {
  const int ea = g.exA[r], e0 = row_exponent(ea) - 5 * (2 * np + 1);
  const int h = min(np, 3), sh = 10 * (np - h);
  const int most = min(4, (g.lower_tiles ? min(g.N, r + 1) : g.N) - c);
  double* cp = g.C + r + (long long)c * g.ldc;
  double old[4];
  if (g.beta != 0.0) {
#pragma unroll
    for (int j = 0; j < 4; j++) old[j] = j < most ? cp[j * g.ldc] : 0.0;
  }
#pragma unroll
  for (int j = 0; j < 4; j++) {
    if (j >= most) break;
    long long W = 0, V = 0;
#pragma unroll
    for (int i = 0; i < MAXPASS; i++) {
      const int x = j == 0 ? q[i].x : j == 1 ? q[i].y : j == 2 ? q[i].z : q[i].w;
      if (i < h) W = W * 1024 + x;
      else if (i < np) V = V * 1024 + x;
    }
    const int eb = g.exB[c + j];
    double v;
    if ((ea & TOP) == TOP || (eb & TOP) == TOP) v = nonfinite_product(ea, eb);
    else v = combine_words(W, sh, V, e0 + row_exponent(eb));
    if (g.alpha != 1.0) v = g.alpha == -1.0 ? -v : v * g.alpha;
    if (g.beta != 0.0) v = fma(g.beta, old[j], v);
    cp[j * g.ldc] = v;
  }
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NTHREADS, 1)
    digit_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                      const __grid_constant__ DgArgs g) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full = (uint64_t*)(smem + TILES * TILE);  // [STEPS], used in the leader
  uint64_t* empty = full + STEPS;                      // [STEPS]
  uint64_t* tfull = empty + STEPS;
  uint64_t* tempty = tfull + 1;  // used in the leader
  uint64_t* drain = tempty + 1;
  uint32_t* tbase_slot = (uint32_t*)(drain + 1);
  volatile int* abort_flag = (volatile int*)(tbase_slot + 1);
  static_assert((STEPS * 2 + 3) * 8 + 8 <= 256, "barriers fit the 256-byte tail");

  const uint32_t rank = cluster_rank();
  const bool lead = rank == 0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int units = dg_units(g);
  const int cid = (int)(blockIdx.x >> 1), ncl = (int)(gridDim.x >> 1);
  const uint16_t BOTH = 0x3;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STEPS; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tfull, 1);
    mbar_init(tempty, 2 * EPI_WARPS);
    mbar_init(drain, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {  // one warp of each CTA allocates the same columns in both
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tbase_slot)),
                 "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  cluster_sync();  // both CTAs' barriers are initialised before either signals the other's
  tc_fence_after();
  const uint32_t tbase = *tbase_slot;
  const uint32_t lead_full = cluster_addr(full, 0);
  const uint64_t ring = desc_sw128(smem);  // tile i is (TILE >> 4) * i further

  if (warp == 0) {
    if (lane == 0) {
      // steps [head, tail) hold their tiles; their counts, four bits a step
      uint32_t head = 0, tail = 0, counts = 0;
      int room = TILES, pos = 0;
      bool ok = true;
      auto release = [&](int site) -> bool {  // waits for the oldest step
        if (!mbar_wait(&empty[head % STEPS], (head / STEPS) & 1, abort_flag, g.err, site, g.wait_ns)) return false;
        room += (counts >> (4 * (head % STEPS))) & 15;
        head++;
        return true;
      };
      // a step: A digits sa and s1 (0: none) and B digit tb of K-step kb
      auto fill = [&](int kb, int ra, int sa, int s1, int rb, int tb) -> bool {
        const int count = (sa > 0) + (s1 > 0) + 1;
        while (room < count || tail - head == STEPS)
          if (!release(41)) return false;
        const int s = tail % STEPS;
        const uint32_t fb = lead_full + 8u * (uint32_t)s;
        if (lead) mbar_expect_tx(&full[s], 2 * count * TILE);  // both CTAs' copies
        auto load = [&](const CUtensorMap* tm, int row, int digit) {
          tma_load_3d_cg2(smem + pos * TILE, tm, kb * ROW, row, digit - 1, fb);
          if (++pos == TILES) pos = 0;
        };
        if (sa > 0) load(&tmA, ra, sa);
        if (s1 > 0) load(&tmA, ra, s1);
        load(&tmB, rb, tb);
        counts = (counts & ~(15u << (4 * s))) | ((uint32_t)count << (4 * s));
        room -= count;
        tail++;
        return true;
      };
#pragma unroll 1
      for (int u = cid; u < units && ok; u += ncl) {
        const Unit U = dg_unit(g, u);
        const int ra = U.mt * 256 + (int)rank * 128, rb = U.nt * 256 + (int)rank * 128;
#pragma unroll 1
        for (int i = U.i0; i < U.i1 && ok; i++) {
          const Pass P = dg_pass(U, i);
#pragma unroll 1
          for (int kb = 0; kb < U.nk && ok; kb++) {
#pragma unroll 1
            for (int t = P.tlo; t <= P.thi && ok; t++)
              ok = fill(U.kb + kb, ra, P.L - t, P.pro && t == P.tlo ? P.L + 1 - t : 0, rb, t);
          }
        }
      }
      // every step filled so far is released by the leader's MMAs: no multicast
      // commit is still on its way to this CTA
      while (ok && head != tail) ok = release(45);
      if (!ok && lead) {  // the leader's barriers track both CTAs' copies of the steps it armed
        const uint64_t deadline = globaltimer_ns() + WAIT_NS;
        for (; head != tail; head++) mbar_drain_until(&full[head % STEPS], (head / STEPS) & 1, deadline);
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && lead) {
      uint32_t step = 0, q = 0;
      int pos = 0;
      bool ok = true, any = false;
#pragma unroll 1
      for (int u = cid; u < units && ok; u += ncl) {
        const Unit U = dg_unit(g, u);
#pragma unroll 1
        for (int i = U.i0; i < U.i1 && ok; i++) {
          const Pass P = dg_pass(U, i);
#pragma unroll 1
          for (int k0 = 0; k0 < U.nk && ok; k0 += P.chunk, q++) {
            {  // both CTAs' epilogues have drained the accumulators
              const uint64_t t0 = globaltimer_ns();
              uint32_t spin = 0;
              while (!mbar_try_wait_cluster(tempty, (q & 1) ^ 1)) {
                const bool every = (spin & 63) == 63, first = spin == 0;  // as in mbar_wait
                spin++;
                if ((every && (*abort_flag || *(volatile int*)g.err)) ||
                    ((every || first) && globaltimer_ns() - t0 > g.wait_ns)) {
                  *abort_flag = 1;
                  atomicCAS(g.err, 0, 42);
                  ok = false;
                  break;
                }
              }
              if (!ok) break;
            }
            tc_fence_after();
            uint32_t use0 = 0, use1 = 0;
            const int k1 = min(U.nk, k0 + P.chunk);
#pragma unroll 1
            for (int kb = k0; kb < k1 && ok; kb++) {
              // the A tile level L + 1 uses next and the step it came with
              uint64_t a1 = 0;
              int from = -1;
#pragma unroll 1
              for (int t = P.tlo; t <= P.thi; t++, step++) {
                const int s = step % STEPS;
                if (!mbar_wait(&full[s], (step / STEPS) & 1, abort_flag, g.err, 43, g.wait_ns)) { ok = false; break; }
                tc_fence_after();
                auto next = [&]() {
                  const uint64_t d = ring + (uint64_t)(pos * (TILE >> 4));
                  if (++pos == TILES) pos = 0;
                  return d;
                };
                const bool has0 = P.L - t >= 1, first = P.pro && t == P.tlo;
                const uint64_t a0 = has0 ? next() : 0;
                if (first) a1 = next();
                const uint64_t b = next();
                if (has0) {
#pragma unroll
                  for (int kk = 0; kk < ROW / 32; kk++) {
                    mma_f8_cg2(tbase, a0 + 2 * kk, b + 2 * kk, DG_IDESC, use0);
                    use0 = 1;
                  }
                }
                if (first || from >= 0) {
#pragma unroll
                  for (int kk = 0; kk < ROW / 32; kk++) {
                    mma_f8_cg2(tbase + 256, a1 + 2 * kk, b + 2 * kk, DG_IDESC, use1);
                    use1 = 1;
                  }
                  if (from >= 0) mma_commit_cg2(&empty[from], BOTH);
                }
                any = true;
                // (the last step's A tile has no further use)
                a1 = a0;
                from = P.has1 && t < P.thi ? s : -1;
                if (from < 0) mma_commit_cg2(&empty[s], BOTH);
              }
              if (!ok) break;
            }
            if (!ok) break;
            mma_commit_cg2(tfull, BOTH);
          }
        }
      }
      if (!ok && any) {
        // all MMAs issued by this thread complete before TMEM is released
        mma_commit_cg2(drain, 0x1);
        mbar_drain(drain, 0);
      }
    }
    __syncwarp();
  } else {
    const int lq = warp & 3;
    const int cbeg = ((warp - 2) >> 2) * EPI_COLS;
    const int row = lq * 32 + lane;
    const uint32_t ta = tbase + ((uint32_t)(lq * 32) << 16) + (uint32_t)cbeg;
    const uint32_t lead_tempty = cluster_addr(tempty, 0);
    // planes as [column / 4][row][column % 4]: sixteen bytes a thread, 512 a warp
    const bool split = g.zsum > 0;
    uint32_t q = 0;
    bool ok = true;
#pragma unroll 1
    for (int u = cid; u < units && ok; u += ncl) {
      const Unit U = dg_unit(g, u);
      const int np = U.i1;
      // (split: the unit's one plane, addressed as level pair i0)
      int4* plane0 = g.planes + cbeg / 4 * 128 + row +
                     (split ? (2 * (size_t)U.slot + rank) * PLANE4 - (ptrdiff_t)U.i0 * PLANE4
                            : (size_t)blockIdx.x * (MAXPASS * PLANE4));
      const int r = U.mt * 256 + (int)rank * 128 + row;
      const int n0 = U.nt * 256 + cbeg;
      const int ncols = max(0, min(EPI_COLS, g.N - n0));
#pragma unroll 1
      for (int i = U.i0; i < np && ok; i++) {
        const Pass P = dg_pass(U, i);
        int4* pl = plane0 + i * PLANE4;
#pragma unroll 1
        for (int k0 = 0; k0 < U.nk; k0 += P.chunk, q++) {
          int okw = 1;
          if (lane == 0) okw = mbar_wait(tfull, q & 1, abort_flag, g.err, 44, g.wait_ns) ? 1 : 0;
          okw = __shfl_sync(0xffffffffu, okw, 0);
          if (!okw) { ok = false; break; }
          tc_fence_after();
#pragma unroll 1
          for (int c0 = 0; c0 < ncols; c0 += 32) {
            uint32_t v[32];
            {
              uint32_t w[32];
              tmem_ld32(ta + c0, v);
              if (P.has1) {
                tmem_ld32(ta + 256 + c0, w);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 32; j++)
                  v[j] = (uint32_t)(exact_f2i(__uint_as_float(v[j])) * 32 + exact_f2i(__uint_as_float(w[j])));
              } else {
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 32; j++) v[j] = (uint32_t)(exact_f2i(__uint_as_float(v[j])) * 32);
              }
            }
#pragma unroll
            for (int j = 0; j < 8; j++) {
              int4* p4 = pl + (c0 / 4 + j) * 128;
              int4 t = make_int4((int)v[4 * j], (int)v[4 * j + 1], (int)v[4 * j + 2], (int)v[4 * j + 3]);
              if (k0 > 0) {
                const int4 o = *p4;
                t = make_int4(t.x + o.x, t.y + o.y, t.z + o.z, t.w + o.w);
              }
              *p4 = t;
            }
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(lead_tempty);
        }
      }
      if (!ok) break;
      if (!split && r < g.M) {
#pragma unroll 1
        for (int c0 = 0; c0 < ncols; c0 += 4) {
          int4 qv[MAXPASS];
#pragma unroll
          for (int i = 0; i < MAXPASS; i++)
            qv[i] = (i < np && U.nk > 0) ? plane0[i * PLANE4 + c0 / 4 * 128] : make_int4(0, 0, 0, 0);
          store_four(g, qv, np, r, n0 + c0);
        }
      }
      __syncwarp();
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();  // the leader's MMAs into both CTAs' TMEM are complete
  tc_fence_after();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(512) : "memory");
  // neither CTA exits while the other may still signal its barriers or copy
  // into its shared memory (see gemm_pair in fgls_ozaki.cu)
  cluster_sync();
  if (*abort_flag) {
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 100000ull) {
    }
  }
}

// Split form: the planes of a tile's level pairs and K parts, four columns of a
// row per thread; the parts are added as integers, exactly.
__global__ void __launch_bounds__(256) digit_combine_kernel(const __grid_constant__ DgArgs g) {
  const int t = blockIdx.x / (2 * PLANE4 / 256);
  const int e = (blockIdx.x % (2 * PLANE4 / 256)) * 256 + threadIdx.x;  // int4 of the tile: rank, column / 4, row
  Unit U;
  dg_tile(g, t, U);
  const int r = U.mt * 256 + e / PLANE4 * 128 + e % 128, c = U.nt * 256 + (e % PLANE4) / 128 * 4;
  if (r >= g.M || c >= (g.lower_tiles ? min(g.N, r + 1) : g.N)) return;
  int4 q[MAXPASS];
  int slot = t * g.zsum;
#pragma unroll
  for (int i = MAXPASS - 1; i >= 0; i--) {
    q[i] = make_int4(0, 0, 0, 0);
    if (i < U.i1) {
      for (int z = 0; z < g.zs[i] && z * g.kper[i] < U.nk; z++) {
        const int4 v = g.planes[(2 * (size_t)(slot + z)) * PLANE4 + e];
        q[i] = make_int4(q[i].x + v.x, q[i].y + v.y, q[i].z + v.z, q[i].w + v.w);
      }
    }
    slot += g.zs[i];
  }
  store_four(g, q, U.i1, r, c);
}

// ------------------------------------------------------------------- digits
constexpr uint64_t DIGIT_BIAS = 16ull * (((1ull << 60) - 1) / 31);  // 16 in every 5-bit field


// |x| 2^(60 - ex) rounded to an integer (|x| < 2^(ex-1)); sign: x's sign bit.
__device__ __forceinline__ unsigned long long to_fixed(double x, int ex, uint32_t& sign) {
  const long long b = __double_as_longlong(x);
  int e = (int)((b >> 52) & 0x7ff);
  unsigned long long m = (unsigned long long)b & 0xfffffffffffffull;
  if (e) m |= 1ull << 52;
  else e = 1;
  const int sh = e - 1015 - ex;  // m 2^sh
  unsigned long long f;
  if (sh >= 0) f = m << min(sh, 11);
  else if (sh > -55) f = (m + (1ull << (-sh - 1))) >> -sh;
  else f = 0;
  sign = (uint32_t)(b >> 32) & 0x80000000u;
  return f;
}
// The four digits of weight 32^-(s+1) of four biased magnitudes, signs applied,
// as E4M3 bytes.  Signs go on the digits because the digits of a magnitude lie
// in [-16, 15], -1/2 on average: cut from signed numbers, the low digits would
// share that mean whatever the signs, and the dropped digit pairs would add up
// over K instead of averaging out.
__device__ __forceinline__ uint32_t digit_word(const uint64_t (&u)[4], const uint32_t (&sg)[4], int s) {
  float f[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const uint32_t d = s == 0 ? (uint32_t)(u[k] >> 55) : (uint32_t)(u[k] >> (55 - 5 * s)) & 31u;
    f[k] = __uint_as_float(__float_as_uint(__fsub_rn(__uint_as_float(0x4B000000u | d), 8388624.0f)) ^ sg[k]);
  }
  const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(f[0], f[1]), __NV_SATFINITE, __NV_E4M3);
  const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(f[2], f[3]), __NV_SATFINITE, __NV_E4M3);
  return lo | (hi << 16);
}
__device__ __forceinline__ int digits_used(unsigned long long bits) {  // of the OR of a row's fixed-point magnitudes
  return bits ? ND - (__ffsll((long long)bits) - 1) / 5 : 0;
}

// One CTA of 256 threads (or one of eight warps, TPR = 32) per row whose
// elements are contiguous in K.  The row is read twice, the second time mostly
// from L2; bound by the writes (twelve bytes an element) and integer issue.
// w > 0: row (i*w + c)*w + d is the product of columns i*w + c and i*w + d.
template <int TPR, bool SIGNS>
__global__ void __launch_bounds__(256) cut_contig_kernel(const double* __restrict__ X, long long ld, int rows, int K,
                                                         int Kpad, int w, uint8_t* __restrict__ D,
                                                         int* __restrict__ ex, int* __restrict__ nd) {
  const int r = blockIdx.x * (256 / TPR) + (int)threadIdx.x / TPR;
  const int l = threadIdx.x % TPR;
  if (TPR == 32 && r >= rows) return;
  const double *x = X + (long long)r * ld, *y = nullptr;
  if (w > 0) {
    x = X + (long long)(r / w) * ld;
    y = X + (long long)(r / (w * w) * w + r % w) * ld;
  }
  auto value = [&](int k) -> double { return y ? x[k] * y[k] : x[k]; };
  int top = 0;
  for (int k = l; k < K; k += TPR)
    top = max(top, (int)((__double_as_longlong(value(k)) >> 52) & 0x7ff));
  __shared__ int stop[8];
  __shared__ unsigned long long sbits[8];
  top = __reduce_max_sync(0xffffffffu, top);
  if (TPR > 32) {
    if ((threadIdx.x & 31) == 0) stop[threadIdx.x >> 5] = top;
    __syncthreads();
    for (int q = 0; q < 8; q++) top = max(top, stop[q]);
  }
  int code = top;
  if (top == TOP) {
    int kinds = 0;  // 1: +inf, 2: -inf, 4: NaN
    for (int k = l; k < K; k += TPR) {
      const long long b = __double_as_longlong(value(k));
      if (((b >> 52) & TOP) == TOP) kinds |= (b & 0xfffffffffffffll) ? 4 : b < 0 ? 2 : 1;
    }
    if (TPR > 32) {
      const int p = __syncthreads_or(kinds & 1), m = __syncthreads_or(kinds & 2), n = __syncthreads_or(kinds & 4);
      kinds = (p ? 1 : 0) | (m ? 2 : 0) | (n ? 4 : 0);
    } else {
      kinds = __reduce_or_sync(0xffffffffu, kinds);
    }
    code |= kinds == 1 ? ALL_PINF : kinds == 2 ? ALL_NINF : 0;
  }
  const int es = row_exponent(top);
  unsigned long long bits = 0;
  int pos = 1, neg = 1;
  for (int g = l; g < Kpad / 4; g += TPR) {
    uint64_t u[4];
    uint32_t sg[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int k = 4 * g + j;
      const double x1 = k < K ? value(k) : 0.0;
      const unsigned long long f = to_fixed(x1, es, sg[j]);
      if (SIGNS && k < K) {
        pos &= x1 > 0.0;
        neg &= x1 < 0.0;
      }
      bits |= f;
      u[j] = f + DIGIT_BIAS;
    }
#pragma unroll
    for (int s = 0; s < ND; s++) *(uint32_t*)(D + ((size_t)s * rows + r) * Kpad + 4 * g) = digit_word(u, sg, s);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) bits |= __shfl_xor_sync(0xffffffffu, bits, o);
  if (TPR > 32) {
    if ((threadIdx.x & 31) == 0) sbits[threadIdx.x >> 5] = bits;
    __syncthreads();
    for (int q = 0; q < 8; q++) bits |= sbits[q];
  }
  if (SIGNS) {
    pos = TPR > 32 ? __syncthreads_and(pos) : (int)__all_sync(0xffffffffu, pos);
    neg = TPR > 32 ? __syncthreads_and(neg) : (int)__all_sync(0xffffffffu, neg);
    code |= pos ? ALL_POS : neg ? ALL_NEG : 0;
  }
  if (l == 0) {
    ex[r] = code;
    atomicMax(nd + (r >> 8), digits_used(bits));
  }
}

// Largest biased exponent of each row of a matrix whose elements are contiguous
// over the rows: 32 rows and a slice of K a CTA, into ex (zero before).
__global__ void __launch_bounds__(256) strided_top_kernel(const double* __restrict__ X, long long ld, int rows, int K,
                                                          int slice, int* __restrict__ ex) {
  __shared__ int stop[8][32];
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const int r = blockIdx.x * 32 + lane, k1 = min(K, ((int)blockIdx.y + 1) * slice);
  int top = 0;
  if (r < rows) {
#pragma unroll 4
    for (int k = blockIdx.y * slice + wp; k < k1; k += 8)
      top = max(top, (int)((__double_as_longlong(X[r + (long long)k * ld]) >> 52) & 0x7ff));
  }
  stop[wp][lane] = top;
  __syncthreads();
  if (wp == 0 && r < rows) {
    for (int q = 1; q < 8; q++) top = max(top, stop[q][lane]);
    atomicMax(ex + r, top);
  }
}

// Digits of such a matrix, ex holding its rows' exponents: 32 x 64 tiles turned
// in shared memory, so that both the loads (256 bytes a warp) and the stores (64
// bytes a row and plane) are coalesced; 32 rows and a slice of K (a multiple of
// 64) a CTA.  (One CTA per 32 rows for all of K: 0.62 ms for 6000 x 6000.)
__global__ void __launch_bounds__(256) cut_strided_kernel(const double* __restrict__ X, long long ld, int rows, int K,
                                                          int Kpad, int slice, uint8_t* __restrict__ D,
                                                          const int* __restrict__ ex, int* __restrict__ nd) {
  __shared__ uint32_t t[ND][32][17];
  __shared__ unsigned long long sbits[8];
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const int r0 = blockIdx.x * 32, r = r0 + lane;
  const double* x = X + r;
  const int es = row_exponent(r < rows ? ex[r] : 0);
  const int kend = min(Kpad, ((int)blockIdx.y + 1) * slice);
  unsigned long long bits = 0;
  for (int k0 = blockIdx.y * slice; k0 < kend; k0 += 64) {
    double v[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {  // two groups of four elements a thread
      const int k = k0 + 8 * wp + j;
      v[j] = (r < rows && k < K) ? x[(long long)k * ld] : 0.0;
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
      uint64_t u[4];
      uint32_t sg[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const unsigned long long f = to_fixed(v[4 * h + j], es, sg[j]);
        bits |= f;
        u[j] = f + DIGIT_BIAS;
      }
#pragma unroll
      for (int s = 0; s < ND; s++) t[s][lane][2 * wp + h] = digit_word(u, sg, s);
    }
    __syncthreads();
    // 12 planes x 32 rows of 16 words: two rows a warp and step
    for (int q = wp * 2 + (lane >> 4); q < ND * 32; q += 16) {
      const int s = q >> 5, rr = q & 31;
      if (r0 + rr < rows)
        *(uint32_t*)(D + ((size_t)s * rows + r0 + rr) * Kpad + k0 + 4 * (lane & 15)) = t[s][rr][lane & 15];
    }
    __syncthreads();
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) bits |= __shfl_xor_sync(0xffffffffu, bits, o);
  if (lane == 0) sbits[wp] = bits;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 0; q < 8; q++) bits |= sbits[q];
    atomicMax(nd + (r0 >> 8), digits_used(bits));
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encoder() {
  static std::atomic<EncodeTiledFn> known{nullptr};
  EncodeTiledFn fn = known.load(std::memory_order_acquire);
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
    known.store(fn, std::memory_order_release);
  }
  return fn;
}

// K-major rows of every digit plane, boxes of 128 digits x 128 rows; rows past
// the matrix are filled with zeros, so no row padding is stored.
cudaError_t digit_map(CUtensorMap* m, const DigitMat& d) {
  EncodeTiledFn enc = encoder();
  if (!enc) return cudaErrorNotSupported;
  cuuint64_t dims[3] = {(cuuint64_t)d.Kpad, (cuuint64_t)d.rows, (cuuint64_t)ND};
  cuuint64_t strides[2] = {(cuuint64_t)d.Kpad, (cuuint64_t)d.Kpad * (cuuint64_t)d.prow};
  cuuint32_t box[3] = {ROW, 128, 1};
  cuuint32_t es[3] = {1, 1, 1};
  const CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, d.d, dims, strides, box, es,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// Clusters of two CTAs of the kernel that the current device holds at once,
// queried once per device; 0 if none can launch.
int dg_clusters() {
  static std::atomic<int> known[64];  // clusters + 1; 0: not queried yet
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  const int v = known[dev].load(std::memory_order_relaxed);
  if (v > 0) return v - 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2);
  cfg.blockDim = dim3(NTHREADS);
  cfg.dynamicSmemBytes = SMEM;
  int n = 0;
  if (cudaFuncSetAttribute(digit_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, (void*)digit_gemm_kernel, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    n = 0;
  }
  known[dev].store(n + 1, std::memory_order_relaxed);
  return n;
}

}  // namespace

struct DigitGemm {
  int clusters = 0;
  int4* planes = nullptr;      // MAXPASS planes a CTA, or one a unit and CTA in the split form (120 MB)
  int* err = nullptr;
  unsigned long long wait_ns = WAIT_NS;
  bool unchecked = false;      // products were launched since digit_gemm_checked
  void* op[2] = {nullptr, nullptr};
  size_t op_bytes[2] = {0, 0};
};

size_t digit_mat_bytes(int rows, int K) {
  const size_t Kpad = (size_t)(K + ROW - 1) / ROW * ROW;
  return (size_t)ND * rows * Kpad + sizeof(int) * ((size_t)rows + (size_t)(rows + 255) / 256) + 512;
}

DigitMat digit_mat_at(void* mem, int rows, int K) {
  DigitMat m;
  m.rows = m.prow = rows;
  m.K = K;
  m.Kpad = (K + ROW - 1) / ROW * ROW;
  m.d = (uint8_t*)mem;
  m.nd = (int*)(m.d + (((size_t)ND * rows * m.Kpad + 255) & ~(size_t)255));
  m.ex = m.nd + (rows + 255) / 256;
  return m;
}

namespace {
cudaError_t cut(cudaStream_t s, const DigitMat& m, const double* X, long long ld, bool kcontig, int w,
                bool signs = false) {
  if (m.rows <= 0 || m.K <= 0 || m.prow != m.rows) return cudaErrorInvalidValue;
  // nd and, behind it, ex
  FGLS_CUDA_TRY(cudaMemsetAsync(m.nd, 0, sizeof(int) * ((m.rows + 255) / 256 + (kcontig ? 0 : m.rows)), s));
  if (!kcontig) {
    // slices of K: about four CTAs an SM
    const int blocks = ceil_div(m.rows, 32);
    const int want = std::max(1, std::min(ceil_div(608, blocks), m.Kpad / 64));
    const int slice = ceil_div(m.Kpad / 64, want) * 64;
    const dim3 grid(blocks, ceil_div(m.Kpad, slice));
    strided_top_kernel<<<grid, 256, 0, s>>>(X, ld, m.rows, m.K, slice, m.ex);
    cut_strided_kernel<<<grid, 256, 0, s>>>(X, ld, m.rows, m.K, m.Kpad, slice, m.d, m.ex, m.nd);
    note_launch();
  } else if (m.K <= 1024)
    (signs ? cut_contig_kernel<32, true> : cut_contig_kernel<32, false>)<<<ceil_div(m.rows, 8), 256, 0, s>>>(
        X, ld, m.rows, m.K, m.Kpad, w, m.d, m.ex, m.nd);
  else
    (signs ? cut_contig_kernel<256, true> : cut_contig_kernel<256, false>)<<<m.rows, 256, 0, s>>>(
        X, ld, m.rows, m.K, m.Kpad, w, m.d, m.ex, m.nd);
  note_launch();
  return cudaGetLastError();
}
}  // namespace

cudaError_t digit_cut(cudaStream_t s, const DigitMat& m, const double* X, long long ld, bool kcontig) {
  return cut(s, m, X, ld, kcontig, 0);
}

cudaError_t digit_cut_signed(cudaStream_t s, const DigitMat& m, const double* X, long long ld) {
  return cut(s, m, X, ld, true, 0, true);
}

cudaError_t digit_cut_products(cudaStream_t s, const DigitMat& m, const double* X, long long ld, int w) {
  return cut(s, m, X, ld, true, w);
}

cudaError_t digit_gemm_create(DigitGemm** out) {
  *out = nullptr;
  const int n = dg_clusters();
  if (n <= 0 || !encoder()) return cudaErrorNotSupported;
  DigitGemm* g = new DigitGemm();
  g->clusters = n;
  cudaError_t r = cudaMalloc(&g->err, sizeof(int));
  if (r == cudaSuccess) r = cudaMemset(g->err, 0, sizeof(int));
  if (r == cudaSuccess) r = cudaDeviceSynchronize();  // the memset ran on the default stream
  if (r != cudaSuccess) {
    digit_gemm_destroy(g);
    return r;
  }
  *out = g;
  return cudaSuccess;
}

void digit_gemm_destroy(DigitGemm* g) {
  if (!g) return;
  void* ptrs[] = {g->planes, g->err, g->op[0], g->op[1]};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  delete g;
}

bool digit_gemm_ready(DigitGemm* g) {
  if (g->planes) return true;
  if (cudaMalloc(&g->planes, sizeof(int4) * (size_t)MAXPASS * PLANE4 * 2 * g->clusters) == cudaSuccess) return true;
  (void)cudaGetLastError();
  g->planes = nullptr;
  return false;
}

int* digit_gemm_error_word(DigitGemm* g) { return g->err; }
bool digit_gemm_unchecked(const DigitGemm* g) { return g && g->unchecked; }
void digit_gemm_checked(DigitGemm* g) { g->unchecked = false; }

void digit_gemm_set_wait_limit(DigitGemm* g, unsigned long long ns) { g->wait_ns = ns ? ns : WAIT_NS; }

cudaError_t digit_mul(DigitGemm* g, cudaStream_t s, const DigitMat& A, const DigitMat& B, double alpha, double beta,
                      double* C, long long ldc, const DigitMulOpts& o) {
  if (A.K != B.K) return cudaErrorInvalidValue;
  if (!digit_gemm_ready(g)) return cudaErrorMemoryAllocation;
  g->unchecked = true;
  CUtensorMap ma, mb;
  FGLS_CUDA_TRY(digit_map(&ma, A));
  FGLS_CUDA_TRY(digit_map(&mb, B));
  DgArgs a;
  a.M = A.rows;
  a.N = B.rows;
  a.tiles_m = ceil_div(A.rows, 256);
  a.tiles_n = ceil_div(B.rows, 256);
  a.lower_tiles = o.c_lower;
  a.a_lower = o.a_lower;
  a.exA = A.ex;
  a.exB = B.ex;
  a.ndA = A.nd;
  a.ndB = B.nd;
  a.alpha = alpha;
  a.planes = g->planes;
  a.err = g->err;
  a.wait_ns = g->wait_ns;
  const int tiles = o.c_lower ? a.tiles_m * (a.tiles_m + 1) / 2 : a.tiles_m * a.tiles_n;
  const int nk_all = A.Kpad / ROW;
  for (int kb = 0; kb < nk_all; kb += K_MAX_STEPS) {
    a.kb0 = kb;
    a.nk = std::min(K_MAX_STEPS, nk_all - kb);
    a.beta = kb > 0 ? 1.0 : beta;
    a.C = C;
    a.ldc = ldc;
    // Few tiles for the clusters: level pairs become units of their own, the
    // larger ones (2 i + 3 stages a K-step) cut along K into parts of at most
    // an even share, as long as the planes of six per cluster hold them.
    a.zsum = 0;
    if (tiles <= SPLIT_TILES * g->clusters) {
      const long long all = (long long)MAXPASS * (MAXPASS + 2) * a.nk * tiles;  // stages of the product
      long long share = std::max(24LL, (all + g->clusters - 1) / g->clusters);
      for (;; share += share / 4) {
        a.zsum = 0;
        for (int i = 0; i < MAXPASS; i++) {
          const int st = (2 * i + 3) * a.nk;
          a.kper[i] = ceil_div(a.nk, std::min<long long>(a.nk, (st + share - 1) / share));
          a.zs[i] = ceil_div(a.nk, a.kper[i]);
          a.zsum += a.zs[i];
        }
        if ((long long)a.zsum * tiles <= (long long)MAXPASS * g->clusters || a.zsum == MAXPASS) break;
      }
      if ((long long)a.zsum * tiles > (long long)MAXPASS * g->clusters) a.zsum = 0;
    }
    const int units = tiles * std::max(1, a.zsum);
    digit_gemm_kernel<<<2 * std::min(g->clusters, units), NTHREADS, SMEM, s>>>(ma, mb, a);
    note_launch();
    if (a.zsum) {
      digit_combine_kernel<<<tiles * (2 * PLANE4 / 256), 256, 0, s>>>(a);
      note_launch();
    }
    FGLS_CUDA_TRY(cudaGetLastError());
  }
  return cudaSuccess;
}

// Estimates in microseconds, from measured products:
//   FP64 kernels: an SM takes 1.0 us per element of K for a 64 x 64 tile (a wave
//     of up to 152; 4096 x 4096 x 5000: 134.6 ms), 0.064 us for a 32 x 8 tile
//     (used below a wave of the others);
//   digits: five launches (60 us), cutting at 6 ps an element, 0.16 us per
//     element of K and wave of 76 tiles of 256 x 256, shared out evenly below a
//     wave, and 50 us a wave for the epilogue beyond it (301 x 74 x 301: 80 us;
//     5000 x 256 x 5000: 0.53 ms; 4096 x 4096 x 64: 0.43 ms, FP64 1.77 ms).
bool digit_gemm_pays(long long M, long long N, long long K) {
  const double k = (double)K;
  const double t64 = (double)((M + 63) / 64) * (double)((N + 63) / 64);
  const double t32 = (double)((M + 31) / 32) * (double)((N + 7) / 8);
  const double t256 = (double)((M + 255) / 256) * (double)((N + 255) / 256);
  const double fp64 = t64 < 152.0 ? 5.0 + 0.064 * k * std::max(1.0, t32 / 152.0) : k * t64 / 152.0;
  const double waves = t256 <= 76.0 ? t256 / 76.0 : std::ceil(t256 / 76.0);
  const double digits = 60.0 + 6e-6 * (double)(M + N) * k + 0.16 * k * waves + (t256 > 76.0 ? 50.0 * waves : 0.0);
  return digits < fp64;
}

namespace {
bool reserve(DigitGemm* g, int q, size_t bytes) {
  if (!digit_gemm_ready(g)) return false;
  if (g->op_bytes[q] >= bytes) return true;
  if (g->op[q]) cudaFree(g->op[q]);
  g->op[q] = nullptr;
  g->op_bytes[q] = 0;
  if (cudaMalloc(&g->op[q], bytes) != cudaSuccess) {
    (void)cudaGetLastError();
    g->op[q] = nullptr;
    return false;
  }
  g->op_bytes[q] = bytes;
  return true;
}
}  // namespace

DigitMat digit_gemm_operand(DigitGemm* g, int q, int rows, int K) {
  if (!reserve(g, q, digit_mat_bytes(rows, K))) return DigitMat();
  return digit_mat_at(g->op[q], rows, K);
}

bool digit_gemm_reserve(DigitGemm* g, int rows, int K) {
  const size_t b = digit_mat_bytes(rows, K);
  return reserve(g, 0, b) && reserve(g, 1, b);
}

bool digit_gemm_trim(DigitGemm* g) {
  if (!g) return false;
  bool held = false;
  for (int q = 0; q < 2; q++) {
    if (g->op[q]) cudaFree(g->op[q]);
    held |= g->op[q] != nullptr;
    g->op[q] = nullptr;
    g->op_bytes[q] = 0;
  }
  return held;
}

bool digit_gemm_release(DigitGemm* g) {
  bool held = digit_gemm_trim(g);
  if (g && g->planes) {
    cudaFree(g->planes);
    g->planes = nullptr;
    held = true;
  }
  return held;
}

cudaError_t digit_dgemm(DigitGemm* g, cudaStream_t s, bool tA, bool tB, int M, int N, int K, double alpha,
                        const double* A, long long lda, const double* B, long long ldb, double beta, double* C,
                        long long ldc, const DigitMulOpts& o) {
  if (g && digit_gemm_pays(M, N, K) && reserve(g, 0, digit_mat_bytes(M, K)) && reserve(g, 1, digit_mat_bytes(N, K))) {
    const DigitMat a = digit_mat_at(g->op[0], M, K), b = digit_mat_at(g->op[1], N, K);
    FGLS_CUDA_TRY(digit_cut(s, a, A, lda, tA));
    FGLS_CUDA_TRY(digit_cut(s, b, B, ldb, !tB));
    return digit_mul(g, s, a, b, alpha, beta, C, ldc, o);
  }
  return dgemm(s, tA, tB, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
}

}  // namespace fgls

// Diagnostic entry point (include/fgls_gb300.h).
extern "C" int fglsgpu_selftest_dgemm(int transA, int transB, int M, int N, int K, double alpha, const double* A,
                                      long long lda, const double* B, long long ldb, double beta, double* C,
                                      long long ldc, int digits, double* ms) {
  using namespace fgls;
  if (M <= 0 || N <= 0 || K <= 0 || !A || !B || !C) return FGLSGPU_EINVAL;
  if (lda < (transA ? K : M) || ldb < (transB ? N : K) || ldc < M) return FGLSGPU_EINVAL;
  cudaStream_t s = nullptr;
  cudaEvent_t ev[2] = {nullptr, nullptr};
  DigitGemm* g = nullptr;
  void* mem[2] = {nullptr, nullptr};
  cudaError_t r = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
  auto chk = [&](cudaError_t e) {
    if (r == cudaSuccess) r = e;
  };
  for (auto& e : ev) chk(cudaEventCreate(&e));
  if (digits) {
    chk(digit_gemm_create(&g));
    if (g && !digit_gemm_ready(g)) chk(cudaErrorMemoryAllocation);
    chk(cudaMalloc(&mem[0], digit_mat_bytes(M, K)));
    chk(cudaMalloc(&mem[1], digit_mat_bytes(N, K)));
  }
  if (r == cudaSuccess) chk(cudaEventRecord(ev[0], s));
  if (r == cudaSuccess && !digits)
    chk(dgemm(s, transA != 0, transB != 0, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc));
  if (r == cudaSuccess && digits) {
    const DigitMat a = digit_mat_at(mem[0], M, K), b = digit_mat_at(mem[1], N, K);
    chk(digit_cut(s, a, A, lda, transA != 0));
    chk(digit_cut(s, b, B, ldb, transB == 0));
    if (r == cudaSuccess) chk(digit_mul(g, s, a, b, alpha, beta, C, ldc));
  }
  if (r == cudaSuccess) chk(cudaEventRecord(ev[1], s));
  if (s) chk(cudaStreamSynchronize(s));
  int herr = 0;
  float t = 0.f;
  if (r == cudaSuccess && g) chk(cudaMemcpy(&herr, digit_gemm_error_word(g), sizeof(int), cudaMemcpyDeviceToHost));
  if (r == cudaSuccess) chk(cudaEventElapsedTime(&t, ev[0], ev[1]));
  if (ms) *ms = t;
  for (void* p : mem)
    if (p) cudaFree(p);
  digit_gemm_destroy(g);
  for (auto e : ev)
    if (e) cudaEventDestroy(e);
  if (s) cudaStreamDestroy(s);
  if (r != cudaSuccess) return FGLSGPU_ECUDA;
  return herr ? FGLSGPU_ETIMEOUT : FGLSGPU_OK;
}
