// Constants and helpers shared by the split-precision kernels (legendre_split.cu,
// legendre_split_pol.cu): tile geometry, the recursion seed and coefficients, the
// pair order of m, the triangular (l, m) table index and the WS row size.
#pragma once
#include "common.cuh"
#include "df64.cuh"
#include "tcgen05.cuh"

#include <cooperative_groups.h>

#include <cmath>

namespace {

constexpr int kRows = 128;          // UMMA M: rows of one parity per l-tile
constexpr int kCols = 128;          // UMMA N: 64 maps x {Re, Im}
constexpr int kGroupMaps = 64;
constexpr int kKStep = 16;          // rings per UMMA
constexpr int kSCRings = 128;       // rings per lambda-digit block
constexpr int kKChunk = 1024;       // rings per CTA (keeps levels 0 and 1 exact)
constexpr int kSlices = 4;
constexpr uint32_t kATileBytes = kRows * kKStep * 2;    // 4 KB per (k-step, digit)
constexpr uint32_t kBTileBytes = kCols * kKStep * 2;    // 4 KB per (k-step, digit)
// Synthesis B tiles carry three more digit planes, d1..d3 times 2^-8 (exact in BF16), so
// the level-4 products fold into the level-3 accumulator.
constexpr int kSynthPlanes = 7;
constexpr uint32_t kSynthBBytes = kSynthPlanes * kBTileBytes;   // 28 KB per l-step
// persistent contractions: eight epilogue warps (two per TMEM lane quarter, one per half of the
// columns), the copy thread's warp and two UMMA warps.  One warp issues about a product per 75
// clocks, the tensor pipe takes one per 63: two warps keep it fed (levels 0 and 3, and 1 and 2).
constexpr int kEpiThreads = 256;
constexpr int kEpiWarps = kEpiThreads / 32;
constexpr int kThreadsG = kEpiThreads + 96;
constexpr int kEmptyExp = -4000;    // column exponent of an all-zero column
// Epilogue staging of the analysis GEMMs: each epilogue warp turns a 32-row x 16-column block
// of results around in shared memory, so that its global stores and reductions go out as
// 128-byte row segments (two rows per instruction) instead of 32 scattered 8-byte values.
// Column j of row r sits at j ^ (r & 15): both the row-wise writes and the column-wise reads
// of a warp touch each bank pair at most twice.
constexpr int kStgWarpDoubles = 32 * 16;
constexpr size_t kStgBytes = (size_t)(kEpiThreads / 32) * kStgWarpDoubles * sizeof(double);
__device__ __forceinline__ int stg_at(int r, int c) { return r * 16 + (c ^ (r & 15)); }

struct RecConst {
  double a, b;
};

__device__ __forceinline__ RecConst rec_coeffs(int l, int m) {
  RecConst c;
  if (l == m) {          // state convention: lambda_m = -b prev = the seed
    c.a = 0.0;
    c.b = -1.0;
    return c;
  }
  const long long L = l, M = m;
  c.a = sqrt((double)((2 * L - 1) * (2 * L + 1)) / (double)(L * L - M * M));
  c.b = sqrt((double)((L - 1) * (L - 1) - M * M) / (double)((2 * L - 3) * (2 * L - 1))) * c.a;
  return c;
}

__device__ __forceinline__ void rec_seed(double sth, double pref, int m, double& v, int& e) {
  int ex;
  double mt = frexp(sth, &ex);
  double rm = 1.0, bm = mt;
  long long re = 0, be = ex;
  for (int k = m; k; k >>= 1) {
    if (k & 1) { rm *= bm; re += be; int t; rm = frexp(rm, &t); re += t; }
    if (k > 1) { bm *= bm; be *= 2; int t; bm = frexp(bm, &t); be += t; }
  }
  rm *= pref;
  { int t; rm = frexp(rm, &t); re += t; }
  if (m & 1) rm = -rm;
  e = (re >= -300) ? 0 : (int)floor((double)(re + 300) / 600.0);
  v = ldexp(rm, (int)(re - 600LL * e));
}

__device__ __forceinline__ int m_of_q(int q, int lmax) {
  return (q & 1) ? lmax - (q >> 1) : (q >> 1);
}
__host__ __device__ __forceinline__ long long tri_off(int m, int lmax) {
  return (long long)m * (2LL * lmax + 3 - m) / 2;
}

// The r-th order (as a pair-order index) of the wave [q0, q1) by ascending m: the work of an
// order falls with m (fewer l, fewer kept rings), so units handed out in this order end on
// small ones.
__device__ __forceinline__ int wave_order(int q0, int q1, int r) {
  const int e0 = q0 + (q0 & 1);                          // first even index: m = q / 2
  const int ne = q1 > e0 ? (q1 - e0 + 1) / 2 : 0;
  if (r < ne) return e0 + 2 * r;
  const int o1 = (q1 & 1) ? q1 - 2 : q1 - 1;             // last odd index: m = lmax - q / 2
  return o1 - 2 * (r - ne);
}

// Work units of a contraction CTA.  The grid has one CTA per unit; a running CTA takes over the
// next unstarted one (cluster launch control) instead of walking a fixed stride, so the units
// spread over the SMs by their actual cost, also while other kernels hold some SMs.  (A fixed
// stride of 152 resonated with the unit order: the busiest SM had 2.0 times the mean work at
// nside 256, and k_tc_gemm's SMs were active 61 % of its time.)  stride > 0 keeps the fixed
// walk, for launches capped to some SMs.  The copy thread asks for the next unit while it loads
// the current one and passes indices through a small ring; -1 ends it.
constexpr int kUq = 4;
struct __align__(16) UnitQueue {
  uint4 resp;
  uint64_t clc, full[kUq], empty[kUq];
  int unit[kUq];
};

__device__ __forceinline__ void uq_init(UnitQueue& q, uint32_t takers /* warps */) {
  tc::mbar_init(&q.clc, 1);
  for (int i = 0; i < kUq; ++i) {
    tc::mbar_init(&q.full[i], 1);
    tc::mbar_init(&q.empty[i], takers);
  }
}
// Copy thread: pass on unit u (the n-th, -1: no more).
__device__ __forceinline__ bool uq_put(UnitQueue& q, uint32_t n, int u, volatile int* abort) {
  if (!tc::mbar_wait(&q.empty[n % kUq], ((n / kUq) & 1) ^ 1, abort)) return false;
  *const_cast<volatile int*>(&q.unit[n % kUq]) = u;
  tc::mbar_arrive(&q.full[n % kUq]);
  return true;
}
// Every other role, by whole warps: the n-th unit, or -1 (also after an expired wait).
__device__ __forceinline__ int uq_take(UnitQueue& q, uint32_t n, volatile int* abort) {
  if (!tc::mbar_wait_warp(&q.full[n % kUq], (n / kUq) & 1, abort)) return -1;
  const int u = *const_cast<volatile int*>(&q.unit[n % kUq]);
  tc::mbar_arrive_warp(&q.empty[n % kUq]);
  return u;
}
// Copy thread: ask for the next unit / the answer to the n-th request (-1: none left).
__device__ __forceinline__ void uq_request(UnitQueue& q) {
  tc::mbar_arrive_expect_tx(&q.clc, 16);
  tc::clc_try_cancel(&q.resp, &q.clc);
}
__device__ __forceinline__ int uq_answer(UnitQueue& q, uint32_t n, volatile int* abort) {
  if (!tc::mbar_wait(&q.clc, n & 1, abort)) return -1;
  const int u = tc::clc_first_cta(&q.resp);
  tc::fence_proxy_async();
  return u;
}
// The whole walk of the copy thread: f(u) loads unit u and returns false on an expired wait.
// On every path the last request has been answered (or its bounded wait has run out).
template <typename F>
__device__ __forceinline__ void uq_walk(UnitQueue& q, int nunits, int stride, volatile int* abort,
                                        F f) {
  int u = blockIdx.x;
  uint32_t n = 0;
  while (true) {
    if (stride == 0) uq_request(q);
    const bool ok = uq_put(q, n, u, abort) && f(u);
    int next;
    if (stride == 0) {
      if (!ok) {
        for (uint32_t it = 0; it < tc::kWaitLimit; ++it)
          if (tc::mbar_try_wait(&q.clc, n & 1)) break;
        return;
      }
      next = uq_answer(q, n, abort);
    } else {
      if (!ok) return;
      next = u + stride < nunits ? u + stride : -1;
    }
    ++n;
    if (next < 0) {
      uq_put(q, n, -1, abort);
      return;
    }
    u = next;
  }
}

// The products of one k-step issued by UMMA warp `side` of a split contraction: ten of level
// a + b <= 3 (digit a of the tiles at ad, digit b of those at bd) into the four level
// accumulators (first: the step starts the accumulation), and with FOLD the three level-4 products
// through the 2^-8 planes of bd, into level 3.  SWAP: bd is the first (M side) operand.
template <bool FOLD, bool SWAP>
__device__ __forceinline__ void split_step(int side, uint32_t tmem, uint64_t ad, uint64_t bd,
                                           uint32_t idesc, bool first) {
  auto mma = [&](int lev, int da, int pb, uint32_t acc) {
    const uint64_t x = tc::umma_desc_add(ad, da * kATileBytes);
    const uint64_t y = tc::umma_desc_add(bd, pb * kBTileBytes);
    tc::umma_bf16_warp(tmem + lev * kCols, SWAP ? y : x, SWAP ? x : y, idesc, acc);
  };
#pragma unroll
  for (int lev = 0; lev <= 3; ++lev) {
    if ((lev == 0 || lev == 3) != (side == 0)) continue;
#pragma unroll
    for (int aa = 0; aa <= lev; ++aa) mma(lev, aa, lev - aa, (!first || aa > 0) ? 1u : 0u);
  }
  if (FOLD && side == 0) {
#pragma unroll
    for (int aa = 1; aa <= 3; ++aa) mma(3, aa, kSlices - 1 + (4 - aa), 1u);
  }
}

// per wave: q0, q1, max l-tiles, max ring K-chunks (analysis), max 128-ring blocks,
// max l-steps, max l K-chunks (synthesis)
constexpr int kWaveInts = 7;

// WS bytes per (m, parity, group): the analysis P tiles (rings) or the synthesis alm tiles
// (l of one parity), whichever is larger
size_t ws_row_bytes(int lmax, int nnorth) {
  const size_t nks = (size_t)(nnorth + kKStep - 1) / kKStep;
  const size_t nkl = (size_t)(lmax / 2 + 1 + kKStep - 1) / kKStep;
  const size_t a = nks * kSlices * kBTileBytes, b = nkl * kSynthBBytes;
  return a > b ? a : b;
}

// Levels 0..3 of one output element (FP32 accumulators, weights 1, 2^-8, 2^-16, 2^-24):
// levels 0 and 1 are exact integers, so their weighted sum is exact as an FP32 (hi, lo)
// pair (two-sum); levels 2 and 3 only touch lo.
__device__ __forceinline__ void combine_levels_pair(uint32_t v0, uint32_t v1, uint32_t v2,
                                                    uint32_t v3, float& hi, float& lo) {
  const float L0 = __uint_as_float(v0);
  const float L1f = __uint_as_float(v1) * 0x1p-8f;
  hi = L0 + L1f;
  const float bv = hi - L0;
  lo = ((L0 - (hi - bv)) + (L1f - bv)) +
       (__uint_as_float(v2) * 0x1p-16f + __uint_as_float(v3) * 0x1p-24f);
}

// The element times (fh + fl) 2^e as an FP64.  The product of the (hi, lo) pair with the
// df64 factor is formed on the FP32 pipe (the high product exact through fmaf, the cross
// terms in the low part, ~2^-46 relative), the power of two goes into the exponent fields
// and one FP64 addition joins the two parts: one FP64 instruction per element instead of
// five (two conversions, an addition, two multiplications).  Exponents below the FP64 range
// give 0, so an empty column (exponent kEmptyExp) writes zeros.
__device__ __forceinline__ double pair_scaled(float hi, float lo, float fh, float fl, int e) {
  const float p = __fmul_rn(hi, fh);
  float q = __fmaf_rn(hi, fh, -p);
  q = __fmaf_rn(hi, fl, q);
  q = __fmaf_rn(lo, fh, q);
  return dd_to_double(p, q, e);
}
__device__ __forceinline__ double levels_scaled(uint32_t v0, uint32_t v1, uint32_t v2,
                                                uint32_t v3, float fh, float fl, int e) {
  float hi, lo;
  combine_levels_pair(v0, v1, v2, v3, hi, lo);
  return pair_scaled(hi, lo, fh, fl, e);
}

// A positive or negative FP64 factor as a df64 pair (setup, once per row).
__device__ __forceinline__ void factor_pair(double x, float& fh, float& fl) {
  fh = __double2float_rn(x);
  fl = __double2float_rn(x - (double)fh);
}

// The slicing kernels read each column twice (its maximum, then its digits) with a few loads in
// flight per thread, so they run at the latency of memory unless many blocks share the work, and a
// wave of a large plan holds only some sixty orders.  The blocks of a cluster (grid z) take one
// part of the summands each and exchange the column maxima through distributed shared memory.
// Size: enough for eight blocks an SM, while a block keeps at least eight k-steps (below that the
// cluster's barriers cost what the shorter loops save).
inline int slice_cluster(long long blocks, int steps) {
  int cl = 1;
  while (cl < 8 && blocks * cl < 8 * 152 && steps >= 16 * cl) cl *= 2;
  return cl;
}
template <class Args>
int launch_slice(void (*k)(Args), dim3 grid, int threads, int cl, cudaStream_t s, const Args& a) {
  if (cl == 1) {
    k<<<grid, threads, 0, s>>>(a);
    FSHT_LAUNCH_CHECK();
    return FSHT_OK;
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  grid.z = cl;
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.stream = s;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = cl;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  FSHT_CUDA_TRY(cudaLaunchKernelEx(&cfg, k, a));
  return FSHT_OK;
}
// The maximum over the cluster of *slot, which every thread of the block sees complete; the block
// must not leave before slice_cluster_done.
__device__ __forceinline__ unsigned long long slice_cluster_max(unsigned long long* slot) {
  auto cl = cooperative_groups::this_cluster();
  cl.sync();
  unsigned long long mx = 0;
  for (unsigned r = 0; r < cl.num_blocks(); ++r)
    mx = max(mx, *cl.map_shared_rank(slot, r));
  return mx;
}
__device__ __forceinline__ void slice_cluster_done() { cooperative_groups::this_cluster().sync(); }

}  // namespace
