// The FP64 Legendre contraction on the 5th-generation tensor cores (tcgen05), at FP64 accuracy.
//
// GB300 runs FP64 FMAs at 1.25 TFLOP/s and BF16 products at 2.4 PFLOP/s, so the plain method's
// contraction (get_plm_recursive + mat2alm / alm2mat, src/sht_core.f90:30-168) is written as
// exact integer products.  Both operands become 62-bit fixed-point numbers against a power-of-two
// scale, cut into eight balanced base-256 digits (|d0| <= 64, |d1..7| <= 128) that BF16 holds
// exactly.  The 36 digit products of level a + b <= 7 run as BF16 UMMAs with FP32 accumulation,
// one accumulator per level: over the 256 summands of a part the sums of levels 0..4 stay
// within 2^24 whatever the digits are (level s >= 1: 256 (2 2^13 + (s - 1) 2^14)), so they are
// exact integers; levels 5..7 carry weights from 2^-40 of the leading product down, where an
// FP32 rounding is far below FP64's.  The epilogue adds every level into one 64-bit integer per
// output element (unit 2^-unit_bits), so no FP64 instruction runs before the last conversion and
// the order of the parts does not matter.
//
// What the fixed point costs: levels 8 and up are dropped, levels 5..7 may round in FP32, and sums
// have a unit of 2^-38 .. 2^-46 of the scale (tc_units.h), all below 2^-44 of the largest operand
// pair; a column has one exponent (spin 2: one for both fields, matrix-form rings: one for a map's
// two rings).  Against long-double sums the rms errors of white, smooth (alm falling as l^-3) and
// constant maps at nside 32..128, lmax 3 nside - 1, are 0.94..1.1 times the FMA kernels' in the
// analyses and 0.5..1.03 times in the syntheses.  Columns that the fixed point cannot hold
// (non-finite, or a maximum beyond 2^+-900) are flagged per (order, 64-map group) and contracted by
// the FMA kernels (legendre_fp64.cu).
//
// Per wave of orders:
//   k_tc_slice      {S, D} phases -> digit tiles and column exponents       (HBM bound)
//   k_tc_lambda     FP64 recursion -> lambda digit tiles, once for all maps (FP64 pipe, 79 %)
//   k_tc_gemm       persistent tcgen05 contraction         (shared-memory and L2 bandwidth)
// and for the synthesis k_tc_slice_alm, k_tc_lambda_T and k_tc_gemm<1, *>.
// nside 512, lmax 1023, 64 maps, each alone: 1.24, 2.8 and 3.6 ms, where the FMA kernel needs 134
// at 82 % of the DFMA rate.
#include "legendre_rec.cuh"
#include "split_common.cuh"
#include "tc_units.h"

#include <algorithm>
#include <cmath>
#include <new>
#include <type_traits>
#include <vector>

namespace {

constexpr int kPlanes = 8;
constexpr uint32_t kPlaneBytes = kRows * kKStep * 2;              // 4 KB: 128 rows x 16 summands
constexpr uint32_t kStepBytes = kPlanes * kPlaneBytes;            // 32 KB per operand and k-step
constexpr uint32_t kHalfBytes = kStepBytes / 2;                   // four planes
constexpr int kPartK = 16;                                        // k-steps per part (256 summands)
constexpr unsigned long long kBias = 0x8080808080808080ull;
constexpr int kFixBits = 62;       // |v| < 2^E becomes |X| < 2^62
constexpr int kMaxExp = 900;       // column maxima beyond 2^+-900 go to the FMA kernels

// v 2^k as a fixed-point integer (truncated), biased so that its eight bytes minus 128 are the
// balanced digits d0 (top byte) .. d7.  Integer instructions only: GB300's FP64 pipe runs two
// operations per clock per SM.  |v 2^k| < 2^62 is the caller's scale.  SUB: v may lie below the
// normal range (elsewhere such a v counts as zero: it is below the scale's last bit).
template <bool SUB = false>
__device__ __forceinline__ unsigned long long fixed_biased(double v, int k) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  const int ex = (int)(b >> 52) & 0x7FF;
  const unsigned long long mant =
      (b & 0xFFFFFFFFFFFFFull) | (!SUB || ex != 0 ? 1ull << 52 : 0ull);
  const int sh = (SUB ? max(ex, 1) : ex) - 1075 + k;
  unsigned long long x = 0;
  if ((SUB || ex != 0) && sh > -53) x = sh >= 0 ? mant << min(sh, 9) : mant >> -sh;
  if ((long long)b < 0) x = 0ull - x;
  return x + kBias;
}

// Digit plane d of eight biased values as eight BF16 (16 bytes): byte b -> 2^23 + b by a byte
// permute, minus 2^23 + 128 (exact), and the high halves of two floats packed.
template <int D>
__device__ __forceinline__ uint4 plane_of(const unsigned long long (&y)[8]) {
  uint32_t f[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t w = D < 4 ? (uint32_t)(y[i] >> 32) : (uint32_t)y[i];
    f[i] = __float_as_uint(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440 | (3 - (D & 3)))) -
                           8388736.f);
  }
  uint4 o;
  o.x = __byte_perm(f[0], f[1], 0x7632);
  o.y = __byte_perm(f[2], f[3], 0x7632);
  o.z = __byte_perm(f[4], f[5], 0x7632);
  o.w = __byte_perm(f[6], f[7], 0x7632);
  return o;
}

__device__ __forceinline__ uint4 neg_bf16(uint4 v) {
  v.x ^= 0x80008000u;
  v.y ^= 0x80008000u;
  v.z ^= 0x80008000u;
  v.w ^= 0x80008000u;
  return v;
}

// The eight planes of one 16-byte core-matrix row (rot: a second copy, negated when neg).
template <bool ROT>
__device__ __forceinline__ void store_planes(unsigned char* dst, unsigned char* rot, bool neg,
                                             const unsigned long long (&y)[8]) {
  auto put = [&](int d, uint4 v) {
    *reinterpret_cast<uint4*>(dst + (size_t)d * kPlaneBytes) = v;
    if (ROT) *reinterpret_cast<uint4*>(rot + (size_t)d * kPlaneBytes) = neg ? neg_bf16(v) : v;
  };
  put(0, plane_of<0>(y));
  put(1, plane_of<1>(y));
  put(2, plane_of<2>(y));
  put(3, plane_of<3>(y));
  put(4, plane_of<4>(y));
  put(5, plane_of<5>(y));
  put(6, plane_of<6>(y));
  put(7, plane_of<7>(y));
}

// Sums leave as FP64 by integer instructions (a conversion and scaling on the FP64 pipe is three
// operations of 15 clocks a warp), combined as integers where two meet, rounded once.
// a 2^e as the nearest FP64, over the whole exponent range.
__device__ __forceinline__ double i64_scaled_any(long long a, int e) {
  unsigned long long u = (unsigned long long)(a < 0 ? -a : a);
  if (u == 0) return 0.0;
  const int lz = __clzll((long long)u);
  u <<= lz;
  const unsigned long long r = (u >> 11) + ((u >> 10) & 1);       // 2^52 .. 2^53
  const int ex = 63 - lz + e + 1023;
  const unsigned long long sign = a < 0 ? 1ull << 63 : 0ull;
  if (ex >= 2047) return __longlong_as_double((long long)(sign | 0x7FF0000000000000ull));
  if (ex <= 0)                                                     // subnormal: u 2^(ex - 12)
    return __longlong_as_double((long long)((ex > -52 ? u >> (12 - ex) : 0ull) | sign));
  return __longlong_as_double(
      (long long)((((unsigned long long)(ex - 1) << 52) + r) | sign));
}
// The same for e of -960 .. 900 (columns beyond 2^+-kMaxExp never come here), without a branch, so
// that several values interleave.
__device__ __forceinline__ double i64_scaled(long long a, int e) {
  const long long s = a >> 63;
  unsigned long long u = (unsigned long long)((a ^ s) - s);
  const int lz = __clzll((long long)u);
  u <<= lz & 63;
  const unsigned long long r = ((u >> 1) + 0x200) >> 10;
  unsigned long long b = r + ((unsigned long long)(unsigned)(e + 1085 - lz) << 52);
  b |= (unsigned long long)s & (1ull << 63);
  return __longlong_as_double((long long)(r ? b : 0ull));
}

// ------------------------------------------------------------------ tables
// Per (l, m): beta, Dm and the exponents (FshtLamRow), D_l = prod a_k carried as the double-
// double product of the exact a_k^2 = (4k^2-1)/(k^2-m^2), so D_l is right to one rounding, and
// beta_l = b_l/(a_l a_{l-1}) = ((l-1)^2-m^2)/(4(l-1)^2-1) to one division.  Spin 2: rows of
// lambda1 and lambda2 themselves (tab2: Dm = 1) and the coefficients a_l, b_l, lam_fact and
// normal_l of the FMA kernels' formulas (ptab).
// Block per m; each thread multiplies out a chunk of l, the chunks are chained by one thread.
constexpr int kTabThreads = 128;

struct TcProd {          // (h + l) 2^e
  double h, l;
  int e;
};
__device__ __forceinline__ TcProd tc_prod(const TcProd& a, double qh, double ql) {
  const double th = a.h * qh;
  double tl = fma(a.h, qh, -th) + (a.h * ql + a.l * qh);
  TcProd r;
  r.h = th + tl;
  r.l = tl - (r.h - th);
  const int t = ilogb(r.h) & ~1;   // an even power of two: the square root stays exact
  r.h = ldexp(r.h, -t);
  r.l = ldexp(r.l, -t);
  r.e = a.e + t;
  return r;
}
__device__ __forceinline__ TcProd tc_prod_a2(const TcProd& a, long long L, long long M) {
  const double num = (double)((2 * L - 1) * (2 * L + 1)), den = (double)(L * L - M * M);
  const double qh = num / den;
  return tc_prod(a, qh, fma(-qh, den, num) / den);
}

__global__ void __launch_bounds__(kTabThreads) k_tc_table(int lmax, FshtLamRow* tab,
                                                          FshtLamRow* tab2, FshtPolRow* ptab) {
  __shared__ TcProd s_p[kTabThreads];
  const int m = blockIdx.x, tid = threadIdx.x;
  const long long M = m, base = tri_off(m, lmax);
  const int n = lmax - m + 1;
  const int chunk = (n + kTabThreads - 1) / kTabThreads;
  const int j0 = min(n, tid * chunk), j1 = min(n, j0 + chunk);
  TcProd p{1.0, 0.0, 0};
  for (int j = max(j0, 1); j < j1; ++j) p = tc_prod_a2(p, m + j, M);
  s_p[tid] = p;
  __syncthreads();
  if (tid == 0) {
    TcProd run{1.0, 0.0, 0};
    for (int t = 0; t < kTabThreads; ++t) {
      const TcProd c = s_p[t];
      s_p[t] = run;                              // the product before chunk t
      run = tc_prod(run, c.h, c.l);
      run.e += c.e;
    }
  }
  __syncthreads();
  p = s_p[tid];
  for (int j = j0; j < j1; ++j) {
    const long long L = m + j;
    if (j > 0) p = tc_prod_a2(p, L, M);
    // square root of the double-double: one Newton correction of the rounded root
    const double s = sqrt(p.h);
    const double dm = s + (fma(-s, s, p.h) + p.l) / (2.0 * s);
    const double bound = sqrt((2.0 * L + 1.0) / (4.0 * M_PI)) * (1.0 + 0x1p-30);
    FshtLamRow r;
    r.beta = j > 1 ? (double)((L - 1) * (L - 1) - M * M) / (double)((2 * L - 3) * (2 * L - 1)) : 0.0;
    r.dm = dm;
    r.dx = p.e / 2;
    r.erow = ilogb(bound / dm) + 1 - r.dx;
    tab[base + j] = r;
    if (!tab2) continue;
    // spin 2: the normalisation N_l of lambda1 and lambda2 = Dm 2^Dx stays out of the tiles too
    // (zero below l = 2)
    const double nl = normal_l((int)L);
    r.dx = nl > 0.0 ? ilogb(nl) : 0;
    r.dm = nl > 0.0 ? ldexp(nl, -r.dx) : 1.0;
    r.erow = ilogb(bound / r.dm) + 1 - r.dx;
    tab2[base + j] = r;
    FshtPolRow c{0.0, 0.0, 0.0, 0.0};
    if (j > 0) {
      const RecConst rc = rec_coeffs((int)L, m);
      c.c1 = rc.a;
      c.c2 = rc.b;
    }
    c.c3 = lam_fact((int)L, m);
    c.c4 = nl;
    ptab[base + j] = c;
  }
}

// ------------------------------------------------------------------ phases -> digits
// grid (q in wave, 4 x group), 128 threads per field: (ring half, map, parity, Re/Im) over a
// quarter (16 maps) of a 64-map group, Re/Im fastest, so that a warp reads whole 32-byte {S, D}
// entries (as in k_slice_phase).  Tile column c = 2 map + comp.  T: every column has its own
// exponent.  Q/U (NF = 2): one exponent per map and order, because lambda1 Q and i lambda2 U
// meet in one integer sum; each field is written plain and as i v = (-Im, Re).
struct TcSliceArgs {
  const double* W[2];    // {S, D} as doubles: [m][ring][map][S|D][Re|Im]
  int kc, nnorth, ngroups, q0, lmax;
  size_t row_bytes;      // per (wave-local q, parity, group, copy)
  const int* ring_i0;
  unsigned char* WS;
  int* EB;
  int* flags;            // per (m, group): four ints, one per 16-map quarter
};

template <int NF>
__global__ void __launch_bounds__(128 * NF) k_tc_slice(TcSliceArgs a) {
  __shared__ unsigned long long s_mx[2 * NF][64];
  const int qi = blockIdx.x, g = blockIdx.y >> 2, quarter = blockIdx.y & 3;
  const int m = m_of_q(a.q0 + qi, a.lmax);
  const int f = NF == 1 ? 0 : (int)(threadIdx.x >> 7);
  const int t = threadIdx.x & 63, half = (threadIdx.x >> 6) & 1;
  const int comp = t & 1, p = (t >> 1) & 1, kl = (t >> 2) + 16 * quarter;
  const int k = g * kGroupMaps + kl;
  const int c = 2 * kl + comp;
  const int i0 = a.ring_i0[m];
  const int K = a.nnorth - i0;
  const int nks = (K + kKStep - 1) / kKStep;
  const int ksh = (nks + 1) / 2;
  const int ks_begin = half ? ksh : 0, ks_end = half ? nks : ksh;
  const int r_begin = ks_begin * kKStep, r_end = min(K, ks_end * kKStep);
  const bool valid = k < a.kc;
  const double* col = a.W[f] + ((((long long)m * a.nnorth + i0) * a.kc + k) * 2 + p) * 2 + comp;
  const long long rstride = (long long)a.kc * 4;
  constexpr unsigned long long kAbs = 0x7FFFFFFFFFFFFFFFull;
  unsigned long long mx = 0;
  if (valid) {
    int r = r_begin;
    for (; r + 8 <= r_end; r += 8) {
      unsigned long long v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        v[u] = (unsigned long long)__double_as_longlong(col[(long long)(r + u) * rstride]) & kAbs;
#pragma unroll
      for (int u = 0; u < 8; ++u) mx = max(mx, v[u]);
    }
    for (; r < r_end; ++r)
      mx = max(mx, (unsigned long long)__double_as_longlong(col[(long long)r * rstride]) & kAbs);
  }
  s_mx[f * 2 + half][t] = mx;
  __syncthreads();
  mx = 0;
  if (NF == 1) {
    mx = max(s_mx[0][t], s_mx[1][t]);
  } else {
#pragma unroll
    for (int h = 0; h < 2 * NF; ++h)
#pragma unroll
      for (int u = 0; u < 4; ++u) mx = max(mx, s_mx[h][(t & ~3) + u]);
  }
  const int ef = (int)(mx >> 52);
  const bool odd_range = mx != 0 && (ef < 1023 - kMaxExp || ef > 1023 + kMaxExp);
  const int E = (mx == 0 || odd_range) ? kEmptyExp : ef - 1022;   // |v| < 2^E
  const int flag = __syncthreads_or(odd_range ? 1 : 0);
  if (threadIdx.x == 0) a.flags[((long long)m * a.ngroups + g) * 4 + quarter] = flag;
  if (f == 0 && !half) a.EB[(((long long)qi * 2 + p) * a.ngroups + g) * kCols + c] = E;
  constexpr int NC = NF == 1 ? 1 : 4;
  unsigned char* base =
      a.WS + (((size_t)(qi * 2 + p) * a.ngroups + g) * NC + 2 * f) * a.row_bytes;
  const int cr = 2 * kl + (comp ^ 1);                     // its column in the i v copy
  unsigned char* dst = base + (c >> 3) * 256 + (c & 7) * 16;
  unsigned char* rot = base + a.row_bytes + (cr >> 3) * 256 + (cr & 7) * 16;
  for (int ts = ks_begin; ts < ks_end; ++ts) {
    double v[kKStep];
#pragma unroll
    for (int u = 0; u < kKStep; ++u) {
      const int r = ts * kKStep + u;
      v[u] = (valid && r < K) ? col[r * rstride] : 0.0;
    }
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      unsigned long long y[8];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        y[j] = E == kEmptyExp ? kBias : fixed_biased(v[hh * 8 + j], kFixBits - E);
      store_planes<NF == 2>(dst + (size_t)ts * kStepBytes + hh * 128,
                            rot + (size_t)ts * kStepBytes + hh * 128, comp == 1, y);
    }
  }
}

// ------------------------------------------------------------------ lambda digits
// The scaled recursion of legendre_split.cu in FP64: mu_l = x mu_{l-1} - beta_l mu_{l-2}, state
// (s1, s2) 2^et brought back to 2^-200 .. 2^200 once per staged block (a step grows it by less
// than 4/3 and shrinks it by at most beta / 2 >= 2^-14).  Two FP64 operations per (l, m, ring)
// bound the kernel, the digits take integer and FP32 instructions beside them.
// Spin 2: the FMA kernels' own recursion (values v 2^(600 e), zero while e < 0) and formulas.
struct TcRing {
  double x;
  double s1, s2;
  int et;
  PolRing pol;
};

__device__ __forceinline__ void tc_seed(TcRing& r, double cth, double sth, double pref, int m,
                                        bool pol) {
  int e, k;
  double v;
  rec_seed(sth, pref, m, v, e);
  r.x = cth;
  r.s2 = 0.0;
  if (pol) {
    r.s1 = v;
    r.et = e;
    r.pol = pol_ring(cth, sth, m);
  } else {
    r.s1 = frexp(v, &k);
    r.et = 600 * e + k;
  }
}

__device__ __forceinline__ int exp_bits(double v) {
  return (int)((unsigned)__double2hiint(v) >> 20) & 0x7FF;
}

__device__ __forceinline__ void tc_rescale(TcRing& r) {
  const int e = max(exp_bits(r.s1), exp_bits(r.s2));
  if (e == 0) return;
  if (e > 1023 + 200) {
    r.s1 *= 0x1p-256;
    r.s2 *= 0x1p-256;
    r.et += 256;
  } else if (e < 1023 - 200) {
    r.s1 *= 0x1p256;
    r.s2 *= 0x1p256;
    r.et -= 256;
  }
}

__device__ __forceinline__ void tc_step(TcRing& r, double beta) {
  const double n = fma(r.x, r.s1, -(beta * r.s2));
  r.s2 = r.s1;
  r.s1 = n;
}

// The values of step j (l = m + j) as biased fixed point against the row exponent (k: 62 minus
// it, plus Dx).
template <int SPIN>
__device__ __forceinline__ void tc_value(TcRing& r, int j, double beta, const FshtPolRow& c,
                                         const PolL& pl, int k, unsigned long long& y1,
                                         unsigned long long& y2) {
  if (SPIN == 2) {
    if (j > 0) rec_step(r.s1, r.s2, r.et, c.c1 * r.x, c.c2);
    y1 = y2 = kBias;
    if (r.et != 0 || __double2hiint(c.c4) == 0) return;
    // N_l is in the row factor: ten FP64 operations a step instead of twelve
    double l1, l2;
    pol_lambda_raw(r.pol, pl, r.s1, r.s2, c.c3, l1, l2);
    y1 = fixed_biased(l1, k);
    y2 = fixed_biased(l2, k);
  } else {
    if (j > 0) tc_step(r, beta);
    y1 = fixed_biased(r.s1, r.et + k);
  }
}

struct TcLamArgs {
  int lmax, nnorth, q0, eag;
  const double* cth;
  const double* sth;
  const double* pref;
  const int* ring_i0;
  const FshtLamRow* tab;
  const FshtPolRow* ptab;
  const long long* lam_off;    // of the layout the kernel writes
  unsigned char* lbuf;
};

constexpr int kTcStride = kSCRings + 2;

// Analysis tiles: rows l of one parity, 16 rings per k-step, one exponent 2^EAG for every row
// (the row factor Dm goes into the epilogue).  grid (q in wave, 128-ring block), 128 threads =
// rings; blocks of 32 (spin 2: 16) l are staged as biased fixed-point values and written out as
// whole core-matrix rows.
template <int SPIN>
__global__ void __launch_bounds__(128) k_tc_lambda(TcLamArgs a) {
  constexpr int NT = SPIN == 2 ? 2 : 1;          // lambda, or lambda1 and lambda2
  constexpr int LB = SPIN == 2 ? 16 : 32;        // l per staged block
  constexpr int RG = LB / 16;                    // groups of eight rows per parity
  __shared__ __align__(16) unsigned long long S[NT][2][LB / 2][kTcStride];
  __shared__ double s_beta[LB];
  __shared__ int s_k[LB];
  __shared__ FshtPolRow s_c[SPIN == 2 ? LB : 1];
  __shared__ PolL s_l[SPIN == 2 ? LB : 1];
  const int q = a.q0 + blockIdx.x;
  const int m = m_of_q(q, a.lmax);
  const int i0 = a.ring_i0[m];
  const int K = a.nnorth - i0;
  const int rb = blockIdx.y;
  if (rb * kSCRings >= K) return;
  const int tid = threadIdx.x;
  const int r = rb * kSCRings + tid;
  const bool valid = r < K;
  const int nks = (K + kKStep - 1) / kKStep;
  const int ntiles = (a.lmax - m + 1 + 2 * kRows - 1) / (2 * kRows);
  unsigned char* base =
      a.lbuf + (size_t)(NT * (a.lam_off[q] - a.lam_off[a.q0])) * kStepBytes;
  const FshtLamRow* tab = a.tab + tri_off(m, a.lmax);
  const FshtPolRow* ptab = SPIN == 2 ? a.ptab + tri_off(m, a.lmax) : nullptr;
  TcRing R{};
  if (valid) tc_seed(R, a.cth[i0 + r], a.sth[i0 + r], a.pref[m], m, SPIN == 2);
  const int nl = a.lmax - m + 1;
  for (int lb = 0; lb < nl; lb += LB) {
    __syncthreads();                             // the previous block has been written out
    if (tid < LB && lb + tid < nl) {
      const FshtLamRow rw = tab[lb + tid];
      s_beta[tid] = rw.beta;
      s_k[tid] = rw.dx + kFixBits - a.eag;
      if (SPIN == 2) {
        s_c[tid] = ptab[lb + tid];
        s_l[tid] = pol_l(m + lb + tid, m);
      }
    }
    __syncthreads();
    if (SPIN == 0) tc_rescale(R);
#pragma unroll 4
    for (int jj = 0; jj < LB; ++jj) {
      const int j = lb + jj;
      unsigned long long y1 = kBias, y2 = kBias;
      if (j < nl && valid)
        tc_value<SPIN>(R, j, s_beta[jj], s_c[SPIN == 2 ? jj : 0], s_l[SPIN == 2 ? jj : 0],
                       s_k[jj], y1, y2);
      S[0][jj & 1][jj >> 1][tid] = y1;
      if (SPIN == 2) S[NT - 1][jj & 1][jj >> 1][tid] = y2;
    }
    __syncthreads();
    const int t = lb / (2 * kRows);
    const int rowt0 = (lb % (2 * kRows)) >> 1;
    for (int u = tid; u < NT * 2 * (LB / 2) * (kSCRings / 8); u += 128) {
      const int r8 = u & 7, khalf = (u >> 3) & 1, ks = (u >> 4) & 7;
      int v = u >> 7;
      const int rg = v % RG;
      v /= RG;
      const int p = v & 1, term = v >> 1;
      const int gks = rb * (kSCRings / kKStep) + ks;
      const int row = rg * 8 + r8;
      if (gks >= nks) continue;
      const unsigned long long* src = &S[term][p][row][ks * kKStep + khalf * 8];
      unsigned long long y[8];
#pragma unroll
      for (int i = 0; i < 8; i += 2) {
        const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(src + i);
        y[i] = w.x;
        y[i + 1] = w.y;
      }
      const int rowt = rowt0 + row;
      unsigned char* tile = base +
                            ((size_t)((term * 2 + p) * ntiles + t) * nks + gks) * kStepBytes +
                            (rowt >> 3) * 256 + khalf * 128 + (rowt & 7) * 16;
      store_planes<false>(tile, nullptr, false, y);
    }
  }
}

// Synthesis tiles: rows = rings, 16 l of one parity per k-step.  The summation index is l, so
// the exponent 2^EA(l) of a row of lambda / Dm moves into the alm digits (k_tc_slice_alm).  A
// thread owns a ring and stores its own 16-byte core-matrix rows.
template <int SPIN>
__global__ void __launch_bounds__(128) k_tc_lambda_T(TcLamArgs a) {
  constexpr int NT = SPIN == 2 ? 2 : 1;
  constexpr int LB = 16;
  __shared__ double s_beta[LB];
  __shared__ int s_k[LB];
  __shared__ FshtPolRow s_c[SPIN == 2 ? LB : 1];
  __shared__ PolL s_l[SPIN == 2 ? LB : 1];
  const int q = a.q0 + blockIdx.x;
  const int m = m_of_q(q, a.lmax);
  const int i0 = a.ring_i0[m];
  const int K = a.nnorth - i0;
  const int rb = blockIdx.y;
  if (rb * kSCRings >= K) return;
  const int tid = threadIdx.x;
  const int r = rb * kSCRings + tid;
  const bool valid = r < K;
  const int nrb = (K + kSCRings - 1) / kSCRings;
  const int nkl = ((a.lmax - m) / 2 + 1 + kKStep - 1) / kKStep;
  unsigned char* base =
      a.lbuf + (size_t)(NT * (a.lam_off[q] - a.lam_off[a.q0])) * kStepBytes + (tid >> 3) * 256 +
      (tid & 7) * 16;
  const FshtLamRow* tab = a.tab + tri_off(m, a.lmax);
  const FshtPolRow* ptab = SPIN == 2 ? a.ptab + tri_off(m, a.lmax) : nullptr;
  TcRing R{};
  if (valid) tc_seed(R, a.cth[i0 + r], a.sth[i0 + r], a.pref[m], m, SPIN == 2);
  const int nl = a.lmax - m + 1;
  for (int lb = 0; lb < nkl * 2 * kKStep; lb += LB) {
    __syncthreads();
    if (tid < LB && lb + tid < nl) {
      const FshtLamRow rw = tab[lb + tid];
      s_beta[tid] = rw.beta;
      s_k[tid] = kFixBits - rw.erow;
      if (SPIN == 2) {
        s_c[tid] = ptab[lb + tid];
        s_l[tid] = pol_l(m + lb + tid, m);
      }
    }
    __syncthreads();
    if (SPIN == 0) tc_rescale(R);
    unsigned long long y[NT][2][8];
#pragma unroll
    for (int jj = 0; jj < LB; ++jj) {
      const int j = lb + jj;
      unsigned long long y1 = kBias, y2 = kBias;
      if (j < nl && valid)
        tc_value<SPIN>(R, j, s_beta[jj], s_c[SPIN == 2 ? jj : 0], s_l[SPIN == 2 ? jj : 0],
                       s_k[jj], y1, y2);
      y[0][jj & 1][jj >> 1] = y1;
      if (SPIN == 2) y[NT - 1][jj & 1][jj >> 1] = y2;
    }
    if (valid) {
      const int kl = lb / (2 * kKStep), half = (lb / LB) & 1;
#pragma unroll
      for (int term = 0; term < NT; ++term)
#pragma unroll
        for (int par = 0; par < 2; ++par)
          store_planes<false>(
              base + ((size_t)((term * 2 + par) * nrb + rb) * nkl + kl) * kStepBytes + half * 128,
              nullptr, false, y[term][par]);
    }
  }
}

// ------------------------------------------------------------------ alm -> digits
// grid (q in wave, group, cluster), 256 threads per field = (half of the block's l steps, comp,
// map): v = a_lm Dm 2^EA(l) with `head` spare bits (tc_units.h), tile column c = 2 map + comp, 16 l
// of one parity per k-step.  T: an exponent per column; E/B (NF = 2): one per map and order, plain
// and i v copies.
struct TcSliceAArgs {
  const double* alm[2];
  int ld, k0, kc, lmax, ngroups, q0, head;
  size_t row_bytes;
  const FshtLamRow* tab;
  unsigned char* WS;
  int* EB;
  int* flags;
};

template <int NF>
__global__ void __launch_bounds__(256 * NF) k_tc_slice_alm(TcSliceAArgs a) {
  __shared__ unsigned long long s_mx[2 * NF][2][2][64];        // [field, half][parity][comp][map]
  __shared__ unsigned long long s_col[2][2][64];               // of the block
  const int qi = blockIdx.x, g = blockIdx.y;
  const int m = m_of_q(a.q0 + qi, a.lmax);
  const int f = NF == 1 ? 0 : (int)(threadIdx.x >> 8);
  const int kl = threadIdx.x & 63, comp = (threadIdx.x >> 6) & 1, half = (threadIdx.x >> 7) & 1;
  const int k = g * kGroupMaps + kl;
  const int c = 2 * kl + comp;
  const bool valid = k < a.kc && !(comp == 1 && m == 0);
  const long long L1 = a.lmax + 1;
  const int nh = 2 * (((a.lmax - m) / 2 + 1 + kKStep - 1) / kKStep);   // blocks of eight l
  const int seg = 2 * (int)blockIdx.z + half, nseg = 2 * (int)gridDim.z;
  const int h0 = nh * seg / nseg, h1 = nh * (seg + 1) / nseg;
  const FshtLamRow* tab = a.tab + tri_off(m, a.lmax);
  const double* col = a.alm[f] + a.k0 + k +
                      (comp == 0 ? (long long)m * L1 + m : (L1 - m) * L1) * a.ld;
  auto cnt_of = [&](int p) { return a.lmax - m - p >= 0 ? (a.lmax - m - p) / 2 + 1 : 0; };
  // bits of |a Dm| 2^EA(l); values too small for the exponent sum count as tiny (the flag of a
  // tiny column maximum sends the whole column to the FMA kernel)
  auto key_of = [&](double w, int ea) -> unsigned long long {
    const unsigned long long b =
        (unsigned long long)__double_as_longlong(w) & 0x7FFFFFFFFFFFFFFFull;
    if ((b >> 52) < 32) return b ? 1ull : 0ull;
    if ((b >> 52) > 2000) return 0x7FF0000000000000ull;
    return b + ((unsigned long long)(long long)ea << 52);
  };
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    unsigned long long mx = 0;
    if (valid) {
      const int e1 = min(cnt_of(p), h1 * 8);
#pragma unroll 8
      for (int idx = h0 * 8; idx < e1; ++idx) {
        const int j = p + 2 * idx;
        const FshtLamRow rw = tab[j];
        mx = max(mx, key_of(__ldg(&col[(long long)j * a.ld]) * rw.dm, rw.erow + rw.dx));
      }
    }
    s_mx[2 * f + half][p][comp][kl] = mx;
  }
  __syncthreads();
  bool flag = false;
  int Ep[2];
  unsigned long long mxp[2];
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    unsigned long long mx = 0;
#pragma unroll
    for (int h = 0; h < 2 * NF; ++h)
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (NF == 2 || (u & 1) == comp) mx = max(mx, s_mx[h][u >> 1][u & 1][kl]);
    if (f == 0 && !half) s_col[p][comp][kl] = mx;
  }
  mxp[0] = slice_cluster_max(&s_col[0][comp][kl]);
  mxp[1] = slice_cluster_max(&s_col[1][comp][kl]);
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    const unsigned long long mx = mxp[p];
    const int ef = (int)(mx >> 52);
    const bool odd_range = mx != 0 && (ef < 1023 - kMaxExp || ef > 1023 + kMaxExp);
    flag |= odd_range;
    Ep[p] = (mx == 0 || odd_range) ? kEmptyExp : ef - 1022 + a.head;
    if (f == 0 && seg == 0) a.EB[(((long long)qi * 2 + p) * a.ngroups + g) * kCols + c] = Ep[p];
  }
  const int any = __syncthreads_or(flag ? 1 : 0);
  if (threadIdx.x < 4 && blockIdx.z == 0)
    a.flags[((long long)m * a.ngroups + g) * 4 + threadIdx.x] = any;
  constexpr int NC = NF == 1 ? 1 : 4;
  const int cr = 2 * kl + (comp ^ 1);
#pragma unroll 1
  for (int p = 0; p < 2; ++p) {
    const int cnt = cnt_of(p), E = p ? Ep[1] : Ep[0];
    unsigned char* base =
        a.WS + (((size_t)(qi * 2 + p) * a.ngroups + g) * NC + 2 * f) * a.row_bytes;
    unsigned char* dst = base + (c >> 3) * 256 + (c & 7) * 16;
    unsigned char* rot = base + a.row_bytes + (cr >> 3) * 256 + (cr & 7) * 16;
    for (int h = h0; h < h1; ++h) {
      double v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int idx = h * 8 + j;
        v[j] = valid && idx < cnt ? __ldg(&col[(long long)(p + 2 * idx) * a.ld]) : 0.0;
      }
      unsigned long long y[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int idx = h * 8 + j;
        y[j] = kBias;
        if (idx < cnt && E != kEmptyExp) {
          const FshtLamRow rw = tab[p + 2 * idx];
          y[j] = fixed_biased(v[j] * rw.dm, rw.erow + rw.dx + kFixBits - E);
        }
      }
      store_planes<NF == 2>(dst + (size_t)(h >> 1) * kStepBytes + (h & 1) * 128,
                            rot + (size_t)(h >> 1) * kStepBytes + (h & 1) * 128, comp == 1, y);
    }
  }
  slice_cluster_done();
}

// ------------------------------------------------------------------ ring transforms
// The DFT of a ring as four real matrix products.  A ring of n = 4 q pixels has its samples at
// (2 j + s) pi / n (s = 1: cap rings and every other belt ring).  Folded about 0 and pi / 2,
//   F_r = sum_j [x_j +- x_{-j} +- x_{pi-j} +- x_{pi+j}] {cos, sin}(r (2 j + s) pi / n),
// even and odd r and cos and sin take one sign pattern each: four q x q products (s = 0: up to
// q + 1) instead of one n x n, 8 q^2 flop per real ring.  Bins r <= n/2 serve every order
// a n +- r, by (-1)^{a s} and a conjugate.  As digit products that is 0.12 ms per map for all
// cap rings of nside 1024 at the tensor rate, and 0.25 measured in tiles of 64 maps (matrices and
// slices included), where Bluestein transforms on the FP64 pipe (two FFTs of 2 n points or more per
// ring) took 0.90 ms.  The belt's power-of-two rings cost q^2 too, and from nside 512 on the FFT is
// the cheaper form there (kDftBeltMax).
// Types: 0 cos r even, 1 cos r odd, 2 sin r even (from 2), 3 sin r odd; row rho of a type is
// r = 2 rho + {0, 1, 2, 1}.
__device__ __forceinline__ int dft_r(int type, int rho) {
  return 2 * rho + (type == 0 ? 0 : type == 2 ? 2 : 1);
}
__device__ __forceinline__ int dft_rows(const FshtDftRing& d, int type) {
  return d.q + ((d.s == 0 && type == 0) ? 1 : 0);
}

// cos(pi t / n) 2^61, t <= n/2, of every class (q, s) (plan creation).
__global__ void k_dft_cos(const FshtDftRing* rings, long long* cosv) {
  const FshtDftRing d = rings[blockIdx.x];
  if (!d.first) return;
  const int n = 4 * d.q;
  for (int t = threadIdx.x; t <= n / 2; t += blockDim.x)
    cosv[d.off_cos + t] = (long long)(cospi((double)t / (double)n) * 0x1p61);
}

struct DftTrigArgs {
  const FshtDftRing* rings;     // of the wave
  const long long* cosv;
  unsigned char* lbuf;
};

// Matrix tiles: rows x 16 summands; forward rows rho and summands j, inverse the other way
// round.  grid (ring of the wave, 4 types x row tile), 256 threads = (row, half of the k-step).
// The class's cosines sit in shared memory; the angle r (2 j + s) mod 2 n moves by a constant
// step along a row.
template <bool INV>
__global__ void __launch_bounds__(256) k_dft_trig(DftTrigArgs a) {
  extern __shared__ long long s_cos[];
  const FshtDftRing d = a.rings[blockIdx.x];
  const int type = blockIdx.y & 3, t = blockIdx.y >> 2;
  if (!d.first || t >= d.nrt) return;
  const int n = 4 * d.q;
  for (int u = threadIdx.x; u <= n / 2; u += 256) s_cos[u] = a.cosv[d.off_cos + u];
  __syncthreads();
  const int r8 = threadIdx.x & 7, half = (threadIdx.x >> 3) & 1, rg = threadIdx.x >> 4;
  const int row = t * kRows + rg * 8 + r8;
  const int nr = dft_rows(d, type), nj = d.q + (d.s == 0 ? 1 : 0);
  const int rows = INV ? nj : nr, ks = INV ? nr : nj;
  unsigned char* dst = a.lbuf +
                       (size_t)(d.off_t + (long long)(type * d.nrt + t) * d.nk) * kStepBytes +
                       rg * 256 + half * 128 + r8 * 16;
  // angle index of summand 0 and its step
  const int r0 = INV ? dft_r(type, 0) : dft_r(type, row);
  const int j0 = INV ? row : 0;
  int step = INV ? 2 * (2 * j0 + d.s) : 2 * r0;
  step %= 2 * n;
  int idx = (int)(((long long)r0 * (2 * j0 + d.s) + (long long)step * (half * 8)) % (2 * n));
  if (type >= 2) idx = (idx + 2 * n - n / 2) % (2 * n);       // sin t = cos(t - pi / 2)
  const int skip = (int)(((long long)step * 8) % (2 * n));
  for (int k = 0; k < d.nk; ++k) {
    unsigned long long y[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      int v = min(idx, 2 * n - idx);                          // 0 .. n
      const bool neg = v > n / 2;
      if (neg) v = n - v;
      long long x = s_cos[v];
      if (neg) x = -x;
      const int kk = k * kKStep + half * 8 + e;
      y[e] = (row < rows && kk < ks) ? (unsigned long long)x + kBias : kBias;
      idx += step;
      if (idx >= 2 * n) idx -= 2 * n;
    }
    idx += skip;
    if (idx >= 2 * n) idx -= 2 * n;
    store_planes<false>(dst + (size_t)k * kStepBytes, nullptr, false, y);
  }
}

struct DftSliceArgs {
  const FshtDftRing* rings;
  int ngroups;
  int head;                     // spare bits of the columns (tc_units.h)
  unsigned char* WS;
  int* EB;                      // per (ring of the wave, group, column)
  // forward: map k of this launch at maps + k map_stride
  const double* maps;
  long long map_stride;
  int nside, nring, cnt;
  // inverse
  const double2* W;
  int kc, nnorth;               // kc: map stride of W; cnt of the maps take part
};
constexpr int kNanExp = kEmptyExp - 1;     // column with a non-finite sample: NaN out

// A fixed-point value without the digit bias.
__device__ __forceinline__ long long fixed_i64(double v, int k) {
  return (long long)(fixed_biased<true>(v, k) - kBias);
}
__device__ __forceinline__ int dft_exp(unsigned long long mx) {
  const int ef = (int)(mx >> 52);
  if (mx == 0) return kEmptyExp;
  return ef == 0x7FF ? kNanExp : max(ef, 1) - 1022;        // (1: below the normal range)
}

// Ring samples -> folded digit tiles.  The ring's samples against the maximum of the map's two
// rings with two bits to spare, so the folds are exact integer sums.
// grid (ring of the wave, MAPS maps), 256 threads = (2 MAPS columns: map, north | south; chunks of
// eight samples).  MAPS = 4: device maps, read twice (the second time from L2), a warp reads 256
// contiguous bytes per map and writes whole 128-byte core matrices.  MAPS = 1: maps in host memory,
// read in place once and kept in shared memory.
template <int MAPS>
__global__ void __launch_bounds__(256) k_dft_slice(DftSliceArgs a) {
  constexpr int COLS = 2 * MAPS, CH = 256 / COLS;
  constexpr bool STAGE = MAPS == 1;
  extern __shared__ double s_x[];              // STAGE: [2][n]
  __shared__ unsigned long long s_mx[8][COLS];
  const FshtDftRing d = a.rings[blockIdx.x];
  const int n = 4 * d.q;
  const int col = threadIdx.x & (COLS - 1), chunk = threadIdx.x / COLS;
  const int map = blockIdx.y * MAPS + (col >> 1), h = col & 1;
  const int ip = a.nring - 1 - d.ring;
  const bool valid = map < a.cnt && !(h == 1 && ip == d.ring);
  const double* x = a.maps + (long long)map * a.map_stride +
                    ring_start(a.nside, h ? ip : d.ring);
  if (STAGE) {
    for (int hh = 0; hh < (ip == d.ring ? 1 : 2); ++hh) {
      const double* g = a.maps + (long long)map * a.map_stride +
                        ring_start(a.nside, hh ? ip : d.ring);
#pragma unroll 4
      for (int j = threadIdx.x; j < n; j += 256) s_x[hh * n + j] = __ldg(&g[j]);
    }
    __syncthreads();
    x = s_x + h * n;
  }
  auto get = [&](int j) { return STAGE ? x[j] : __ldg(&x[j]); };
  unsigned long long mx = 0;
  if (valid)
    for (int j0 = chunk * 8; j0 < n; j0 += 8 * CH) {
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (j0 + e < n)
          mx = max(mx, (unsigned long long)__double_as_longlong(get(j0 + e)) &
                           0x7FFFFFFFFFFFFFFFull);
    }
  // one exponent for the map's two rings: their sum and difference are formed as integers
  mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
#pragma unroll
  for (int o = COLS; o < 32; o *= 2) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) < COLS) s_mx[threadIdx.x >> 5][col] = mx;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; ++w) mx = max(mx, s_mx[w][col]);
  const int E = dft_exp(mx);
  const bool live = valid && E > kEmptyExp;
  const int g = map >> 6, c = 2 * (map & 63) + h;
  if (map >= a.cnt) return;
  if (chunk == 0)
    a.EB[((long long)blockIdx.x * a.ngroups + g) * kCols + c] =
        E > kEmptyExp ? E + 2 + a.head : E;
  const int nj = d.q + (d.s == 0 ? 1 : 0);
  unsigned char* dst = a.WS + (size_t)(d.off_c * a.ngroups) * kStepBytes +
                       (size_t)g * d.nk * kStepBytes + (c >> 3) * 256 + (c & 7) * 16;
  const size_t tstride = (size_t)a.ngroups * d.nk * kStepBytes;
  const int kf = kFixBits - 2 - a.head - E;
  for (int hc = chunk; hc < 2 * d.nk; hc += CH) {
    unsigned long long y[4][8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int j = hc * 8 + e;
      long long x0 = 0, x1 = 0, x2 = 0, x3 = 0;
      if (live && j < nj) {
        const bool lo = d.s == 0 && j == 0, hi = d.s == 0 && j == d.q;   // samples on an axis
        x0 = fixed_i64(get(j), kf);
        if (!lo) x1 = fixed_i64(get(n - d.s - j), kf);
        if (!hi) x2 = fixed_i64(get(n / 2 - d.s - j), kf);
        if (!lo && !hi) x3 = fixed_i64(get(n / 2 + j), kf);
      }
      const long long u = x0 + x1, u2 = x2 + x3, v = x0 - x1, v2 = x2 - x3;
      y[0][e] = (unsigned long long)(u + u2) + kBias;
      y[1][e] = (unsigned long long)(u - u2) + kBias;
      y[2][e] = (unsigned long long)(v - v2) + kBias;
      y[3][e] = (unsigned long long)(v + v2) + kBias;
    }
#pragma unroll
    for (int ty = 0; ty < 4; ++ty)
      store_planes<false>(dst + ty * tstride + (size_t)(hc >> 1) * kStepBytes + (hc & 1) * 128,
                          nullptr, false, y[ty]);
  }
}

// c (-1)^{a s} sums of G over the orders of bin r: x = sum_r A_r cos - B_r sin.  Most bins have
// the orders r and n - r at most, loaded without a loop so that several bins are in flight.
__device__ __forceinline__ double2 dft_bin(const double2* __restrict__ g, long long stride_m,
                                           const FshtDftRing& d, int r) {
  const int n = 4 * d.q;
  const bool self = r == 0 || 2 * r == n;
  const double2 zero = make_double2(0.0, 0.0);
  const double2 z0 = r <= d.mtop ? g[(long long)r * stride_m] : zero;
  const double2 z1 = !self && n - r <= d.mtop ? g[(long long)(n - r) * stride_m] : zero;
  const double w0 = r == 0 ? 1.0 : 2.0, w1 = d.s ? -2.0 : 2.0;
  double2 v = make_double2(fma(w1, z1.x, w0 * z0.x), fma(-w1, z1.y, w0 * z0.y));
  double sg = w1;
  for (int m = n + r; m <= d.mtop; m += n) {         // a n + r and (a + 1) n - r
    const double2 z = g[(long long)m * stride_m];
    v.x = fma(sg, z.x, v.x);
    v.y = fma(sg, z.y, v.y);
    if (d.s) sg = -sg;
    const int m1 = m + n - 2 * r;
    if (!self && m1 <= d.mtop) {
      const double2 y = g[(long long)m1 * stride_m];
      v.x = fma(sg, y.x, v.x);
      v.y = fma(-sg, y.y, v.y);
    }
  }
  return v;
}

// {G_N, G_S} -> digit tiles of A (cos types) and B (sin types).  grid (ring of the wave, 16 maps),
// lanes = columns (map, north | south): a warp reads 512 contiguous bytes per order.
__global__ void __launch_bounds__(256) k_dft_slice_inv(DftSliceArgs a) {
  __shared__ unsigned long long s_mx[8][32];
  const FshtDftRing d = a.rings[blockIdx.x];
  const int n = 4 * d.q;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int map = blockIdx.y * 16 + (lane >> 1), h = lane & 1;
  const bool valid = map < a.cnt && !(h == 1 && d.ring == a.nnorth - 1);
  const long long stride_m = (long long)a.nnorth * a.kc * 2;
  const double2* g = a.W + ((long long)d.ring * a.kc + (map < a.cnt ? map : 0)) * 2 + h;
  unsigned long long mx = 0;
  if (valid)
#pragma unroll 4
    for (int r = warp; r <= n / 2; r += 8) {
      const double2 v = dft_bin(g, stride_m, d, r);
      const unsigned long long bx =
          (unsigned long long)__double_as_longlong(v.x) & 0x7FFFFFFFFFFFFFFFull;
      const unsigned long long by =
          (unsigned long long)__double_as_longlong(v.y) & 0x7FFFFFFFFFFFFFFFull;
      mx = max(mx, max(bx, by));
    }
  s_mx[warp][lane] = mx;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; ++w) mx = max(mx, s_mx[w][lane]);
  const int E = dft_exp(mx);
  const bool live = valid && E > kEmptyExp;
  const int grp = map >> 6, c = 2 * (map & 63) + h;
  if (map >= a.cnt) return;
  if (warp == 0)
    a.EB[((long long)blockIdx.x * a.ngroups + grp) * kCols + c] = E > kEmptyExp ? E + a.head : E;
  unsigned char* dst = a.WS + (size_t)(d.off_c * a.ngroups) * kStepBytes +
                       (size_t)grp * d.nk * kStepBytes + (c >> 3) * 256 + (c & 7) * 16;
  const size_t tstride = (size_t)a.ngroups * d.nk * kStepBytes;
  for (int hc = warp; hc < 2 * d.nk; hc += 8)
#pragma unroll 1
    for (int ty = 0; ty < 4; ++ty) {
      const int nr = dft_rows(d, ty);
      unsigned long long y[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int rho = hc * 8 + e;
        y[e] = kBias;
        if (live && rho < nr) {
          const double2 v = dft_bin(g, stride_m, d, dft_r(ty, rho));
          y[e] = fixed_biased<true>(ty < 2 ? v.x : v.y, kFixBits - a.head - E);
        }
      }
      store_planes<false>(dst + ty * tstride + (size_t)(hc >> 1) * kStepBytes + (hc & 1) * 128,
                          nullptr, false, y);
    }
}

// ------------------------------------------------------------------ contraction
// Persistent, one CTA per SM, units from the queue of split_common.cuh.  A unit is a 128-column
// (64 maps x Re/Im, the UMMA M side = TMEM lanes) x N-row tile: N <= 128 l-rows of one parity
// (DIR 0, analysis) or rings (DIR 1, synthesis), over one or two phases of one or two segments:
//   DIR 0          one phase;  spin 2: lambda1 against the field, lambda2 against i x the other
//   DIR 1          phase 0 gives A, phase 1 gives B', north = A + B', south = A - B':
//                  T: even l, then odd l; Q/U: (lambda1 even, lambda2 odd), then (lambda1 odd,
//                  lambda2 even), since lambda1 keeps (-1)^(l-m) and lambda2 takes the opposite
//   DIR 2, 3       ring transforms, forward and inverse (below)
// Each part of <= kPartK k-steps runs two passes through the four 128-column TMEM accumulators:
// levels 0..3 (digit planes 0..3) and levels 4..7 (all planes).  The slots form two pairs, each
// with a UMMA warp and barriers of its own: pair 0 finishes its smaller share first and is drained
// into the 64-bit integers while the products of pair 1 still run.  Shorter parts cost more passes:
// 11 k-steps 5 % more, 8 k-steps 11 %.  One lane copies (16 KB of each operand per stage).
// What bounds it (nside 512, lmax 1023, 64 maps): shared memory, 328 KB a k-step at 128 bytes a
// clock = 2624 clocks against 2304 on the tensor pipe, and the copies, 96 KB a k-step (8.4 TB/s
// over all SMs, about half of it from HBM at 55 % of its rate); tensor pipe 65 % active.
// The map columns are on the lanes, so a warp's alm stores are two 128-byte segments and its
// phase-matrix stores whole {Re, Im} pairs, with no staging through shared memory.
// Sixteen epilogue warps (four per TMEM lane quarter, one per 32 accumulator columns: 32 64-bit
// sums a thread), then the copy thread's warp and two UMMA warps.  With eight warps and 64 sums a
// thread the drains and the output ran at the latency of two warps per scheduler.
constexpr int kTcEpi = 512, kTcEpiWarps = kTcEpi / 32;
constexpr int kTcAcc = 32;
constexpr int kTcThreads = kTcEpi + 96;
constexpr int kTcStages = 6;
constexpr uint32_t kTcStageBytes = 2 * kHalfBytes;              // 32 KB
constexpr size_t kTcSmem = (size_t)kTcStages * kTcStageBytes;

struct TcGemmArgs {
  int lmax, nnorth, ngroups, q0, q1, ntmax, nunits;
  int nfield, field0;          // spin 2: fields of this call (E/Q = 0, B/U = 1)
  int accumulate, unit_bits, eag;
  size_t row_bytes;
  const int* ring_i0;
  const long long* lam_off;
  const FshtLamRow* tab;
  const unsigned char* lbuf;
  const unsigned char* WS;
  const int* EB;
  const int* flags;
  double* out[2];              // DIR 0: alm of T/E, B; DIR 1: phase matrices of T/Q, U
  int ld, k0, kc;
  double pa;                   // DIR 0: factor of the sums
  int* err;
  // ring transforms (DIR 2, 3): the rings of the wave, map k_off + k of W / map k of maps
  const FshtDftRing* rings;
  long long map_stride;
  int nside, nring, k_off, w_kc;
};

struct __align__(8) TcSmemHdr {
  uint64_t full[kTcStages], empty[kTcStages], tfull[2], tempty[2], fin;
  uint32_t tmem;
  int abort;
};

struct TcUnit {
  int g, field, p, t, qi, m, nk, nt, row0, nrows, N;
  FshtDftRing d;               // DIR 2, 3
};

template <int DIR, int SPIN>
__device__ __forceinline__ TcUnit tc_unit(const TcGemmArgs& a, int u) {
  TcUnit w;
  w.g = u % a.ngroups;
  int r = u / a.ngroups;
  w.field = 0;
  if (DIR >= 2) {
    w.p = 0;
    if (DIR == 2) {
      w.p = r & 3;                                         // type
      r >>= 2;
    }
    w.t = r % a.ntmax;
    w.qi = r / a.ntmax;
    w.d = a.rings[w.qi];
    w.m = w.d.ring;
    w.nt = w.d.nrt;
    w.row0 = w.t * kRows;
    if (DIR == 2) {
      // rows rho whose bin r some kept order reaches
      const int r0 = dft_r(w.p, 0);
      const int need = w.d.mtop >= r0 ? (w.d.mtop - r0) / 2 + 1 : 0;
      w.nrows = max(0, min(kRows, min(dft_rows(w.d, w.p), need) - w.row0));
      w.N = (w.nrows + 15) & ~15;
    } else {
      w.nrows = max(0, min(kRows, w.d.q + (w.d.s == 0 ? 1 : 0) - w.row0));
      w.N = (2 * min(kGroupMaps, a.kc - w.g * kGroupMaps) + 15) & ~15;   // map columns
    }
    w.nk = w.nrows > 0 ? w.d.nk : 0;
    return w;
  }
  if (SPIN == 2) {
    w.field = a.field0 + r % a.nfield;
    r /= a.nfield;
  }
  w.p = 0;
  if (DIR == 0) {
    w.p = r & 1;
    r >>= 1;
  }
  w.t = r % a.ntmax;
  w.qi = wave_order(a.q0, a.q1, r / a.ntmax) - a.q0;
  w.m = m_of_q(a.q0 + w.qi, a.lmax);
  const int i0 = a.ring_i0[w.m];
  const int K = a.nnorth - i0;
  if (DIR == 0) {
    w.nt = (a.lmax - w.m + 1 + 2 * kRows - 1) / (2 * kRows);
    w.row0 = w.m + w.t * 2 * kRows + w.p;                // l of row 0
    w.nrows = w.row0 <= a.lmax ? min(kRows, (a.lmax - w.row0) / 2 + 1) : 0;
    w.nk = w.nrows > 0 ? (K + kKStep - 1) / kKStep : 0;
  } else {
    w.nt = (K + kSCRings - 1) / kSCRings;
    w.row0 = i0 + w.t * kSCRings;                        // ring of row 0
    w.nrows = max(0, min(kRows, K - w.t * kSCRings));
    w.nk = w.nrows > 0 ? ((a.lmax - w.m) / 2 + 1 + kKStep - 1) / kKStep : 0;
  }
  w.N = (w.nrows + 15) & ~15;
  return w;
}

// The products of levels L and L + 1 for one k-step into the slot pair at `slot`.  Neighbouring
// digit planes of the second operand are neighbours in shared memory and the two levels' slots in
// TMEM, so where the tile is wide one 256-column product a_i x {b_(L-i), b_(L+1-i)} serves both
// levels and reads a_i once: 36 products of 128 columns read 288 KB of shared memory a k-step
// beside the 96 KB that the copies write (3072 clocks at 128 bytes a clock against 2304 on the
// tensor pipe), 14 wide and 8 narrow ones 232.
// (The two halves of an operand's planes lie in different stages: no pair spans planes 3 and 4.)
constexpr int kWideN = 96;
template <int L, class F>
__device__ __forceinline__ void tc_products(uint32_t slot, const F& plane, uint32_t id1, bool wide,
                                            bool accumulate) {
  const uint32_t id2 = tc::umma_idesc_bf16(kRows, 2 * kCols);
  if (wide) {
#pragma unroll
    for (int i = 0; i <= L + 1; ++i) {
      const int b = L - i;
      const uint32_t acc = accumulate || i > 0 ? 1u : 0u;
      if (b >= 0 && b != 3) {
        tc::umma_bf16_warp(slot, plane(i, false), plane(b, true), id2, acc);
      } else {
        if (b >= 0) tc::umma_bf16_warp(slot, plane(i, false), plane(b, true), id1, acc);
        tc::umma_bf16_warp(slot + kCols, plane(i, false), plane(b + 1, true), id1, acc);
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i <= L + 1; ++i) {
      const uint32_t acc = accumulate || i > 0 ? 1u : 0u;
      if (i <= L) tc::umma_bf16_warp(slot, plane(i, false), plane(L - i, true), id1, acc);
      tc::umma_bf16_warp(slot + kCols, plane(i, false), plane(L + 1 - i, true), id1, acc);
    }
  }
}

// Segment sg of phase ph: its column tiles, lambda tiles and sign.
template <int DIR, int SPIN>
__device__ __forceinline__ void tc_segment(const TcGemmArgs& a, const TcUnit& w, int ph, int sg,
                                           const unsigned char*& cols, const unsigned char*& rows,
                                           int& sign) {
  constexpr int NT = SPIN == 2 ? 2 : 1, NC = SPIN == 2 ? 4 : 1;
  if (DIR >= 2) {
    const int type = DIR == 2 ? w.p : ph;
    sign = 1;
    cols = a.WS + (size_t)(w.d.off_c * a.ngroups + (long long)(type * a.ngroups + w.g) * w.d.nk) *
                      kStepBytes;
    rows = a.lbuf + (size_t)(w.d.off_t + (long long)(type * w.d.nrt + w.t) * w.d.nk) * kStepBytes;
    return;
  }
  const int par = DIR == 0 ? (w.p ^ sg) : (ph ^ sg);
  const int lpar = DIR == 0 ? w.p : par;                 // parity of the lambda rows / l
  int copy = 0;
  sign = 1;
  if (SPIN == 2) {
    copy = sg == 0 ? 2 * w.field : 2 * (1 - w.field) + 1;
    if (DIR == 0)
      sign = (sg == 1 && w.field == 1) ? -1 : 1;
    else
      sign = (sg == 1 && w.field == 1) ? 1 : -1;
  }
  cols = a.WS + (((size_t)(w.qi * 2 + par) * a.ngroups + w.g) * NC + copy) * a.row_bytes;
  rows = a.lbuf +
         ((size_t)(NT * (a.lam_off[a.q0 + w.qi] - a.lam_off[a.q0])) +
          (size_t)((sg * 2 + lpar) * w.nt + w.t) * w.nk) * kStepBytes;
}

// acc += the level sums of two neighbouring slots (levels 2 PAIR and 2 PAIR + 1), 32 columns per
// thread, times sg.  Integers come out of the mantissa of L + 1.5 2^23 (the conversion instruction
// took three times as long, with the UMMA warps waiting), and the two levels are joined in 32 bits
// first, so a pair costs one 64-bit multiply-add, which runs at about an eighth of the FP32 rate:
//   PAIR 0, 1, 2: t = 256 n_a + n_b with weight 2^wt of level b; PAIR 3: the rounded
//   2^(unit_bits - 48) (L_6 + 2^-8 L_7).
// The constants that the mantissa trick leaves in t (kBias2, kMagic) stay in acc until the end of
// the unit.  |L| < 2^22 holds for levels 0 and 1 over 256 summands; larger sums of the others need
// extreme digits throughout and take the conversion.
constexpr uint32_t kMagic = 0x4B400000u, kBias2 = 0x8B400000u;   // kBias2 = 257 kMagic mod 2^32
template <int PAIR>
__device__ __forceinline__ void tc_drain(uint32_t ta, uint32_t tb, int nrow, float sg,
                                         int unit_bits, unsigned long long (&acc)[kTcAcc]) {
  const int wt = unit_bits - 16 * PAIR - 8;                      // of the second level
  const float f6 = sg * __int_as_float((127 + unit_bits - 48) << 23), f7 = f6 * 0x1p-8f;
  const uint32_t mul = PAIR == 3 ? 1u : 1u << (wt >= 32 ? wt - 32 : wt);
  const bool hi = PAIR == 0 && wt >= 32;
#pragma unroll
  for (int c = 0; c < kTcAcc; c += 8) {
    if (c >= nrow) break;
    uint32_t va[8], vb[8];
    tc::tmem_ld8(ta + c, va);
    tc::tmem_ld8(tb + c, vb);
    tc::tmem_wait_ld();
    auto A = [&](int j) { return __uint_as_float(va[j]); };
    auto B = [&](int j) { return __uint_as_float(vb[j]); };
    bool big = false;
    if (PAIR > 0) {
      float mx = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) mx = fmaxf(mx, fmaxf(fabsf(A(j)), fabsf(B(j))));
      big = __any_sync(0xffffffffu, mx >= 0x1p22f);
    }
    auto put = [&](int j, uint32_t t) {
      if (hi)
        acc[c + j] = ((unsigned long long)((uint32_t)(acc[c + j] >> 32) + t * mul) << 32) |
                     (uint32_t)acc[c + j];
      else
        acc[c + j] += (unsigned long long)t * mul;
    };
    if (!big) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (PAIR == 3)
          put(j, __float_as_uint(fmaf(A(j), f6, B(j) * f7) + 12582912.f));
        else
          put(j, __float_as_uint(fmaf(A(j), sg, 12582912.f)) * 256u +
                     __float_as_uint(fmaf(B(j), sg, 12582912.f)));
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (PAIR == 3) {
          acc[c + j] += (unsigned long long)(__float2ll_rn(fmaf(A(j), f6, B(j) * f7)) +
                                             (long long)kMagic);
        } else {
          const long long t = (long long)__float2int_rn(A(j) * sg) * 256 + __float2int_rn(B(j) * sg);
          acc[c + j] += (unsigned long long)(t + (long long)kBias2) * mul;
        }
      }
    }
  }
}

// Finished sums n0 .. n0 + cnt - 1 of column c (TMEM lane) of the unit's tile (DIR 3: matrix row
// c, map columns n); every lane of the warp calls it.  What is read back is read before anything
// is written, so the loads are in flight together.
template <int DIR, int SPIN, int kOut>
__device__ __forceinline__ void tc_out(const TcGemmArgs& a, const TcUnit& w, int ph, bool store,
                                       int c, int n0, int cnt, int map, int eb, int e,
                                       const long long (&sum)[kOut],
                                       const double* fac) {
  const int comp = c & 1;
  double v[kOut];
  if (DIR == 0) {
    if (!store) return;
    const long long L1 = a.lmax + 1;
    const long long row = comp == 0 ? (long long)w.m * L1 + w.row0 + 2 * n0
                                    : (L1 - w.m) * L1 + (w.row0 - w.m) + 2 * n0;
    double* d = a.out[SPIN == 2 ? w.field : 0] + row * a.ld + a.k0 + map;
    const long long ds = 2LL * a.ld;
    // (column exponents beyond 2^+-kMaxExp never come here)
#pragma unroll
    for (int j = 0; j < kOut; ++j) v[j] = i64_scaled(sum[j], e) * fac[j];
    if (a.accumulate) {
      double old[kOut];
#pragma unroll
      for (int j = 0; j < kOut; ++j) old[j] = j < cnt ? d[j * ds] : 0.0;
#pragma unroll
      for (int j = 0; j < kOut; ++j) v[j] += old[j];
    }
#pragma unroll
    for (int j = 0; j < kOut; ++j)
      if (j < cnt) d[j * ds] = v[j];
  } else if (DIR == 1) {
    if (!store) return;
    double* d = a.out[SPIN == 2 ? w.field : 0] +
                (((long long)w.m * a.nnorth + w.row0 + n0) * a.kc + map) * 4 + comp;
    const long long ds = (long long)a.kc * 4;
    if (ph == 0) {                   // A waits, as its integer, in the slot of the same thread
#pragma unroll
      for (int j = 0; j < kOut; ++j)
        if (j < cnt) d[j * ds] = __longlong_as_double(sum[j]);
    } else {
#pragma unroll
      for (int j = 0; j < kOut; ++j) v[j] = j < cnt ? d[j * ds] : 0.0;
      double x[kOut];
#pragma unroll
      for (int j = 0; j < kOut; ++j) {
        const long long A = __double_as_longlong(v[j]);
        v[j] = i64_scaled(A + sum[j], e);
        x[j] = i64_scaled(A - sum[j], e);
      }
#pragma unroll
      for (int j = 0; j < kOut; ++j)
        if (j < cnt) {
          d[j * ds] = v[j];
          d[j * ds + 2] = x[j];
        }
    }
  } else if (DIR == 2) {
    // {S, D} = F_N +- F_S from the lane pair (the map's north and south), then every kept order
    // a n +- r of bin r
    const int nr = 4 * w.d.q, cmp = w.p >= 2;
    double* d = a.out[0] + (((long long)w.m * a.w_kc + a.k_off + map) * 2 + comp) * 2;
    const long long ms = (long long)a.nnorth * a.w_kc * 4;
    unsigned long long y[kOut];                    // bits of the values, Im F = -(sin sum)
#pragma unroll
    for (int j = 0; j < kOut; ++j) {
      const long long o = __shfl_xor_sync(0xffffffffu, sum[j], 1);
      const long long t = comp == 0 ? sum[j] + o : o - sum[j];
      y[j] = (unsigned long long)__double_as_longlong(i64_scaled_any(cmp ? -t : t, e));
      if (eb == kNanExp) y[j] = 0x7FF8000000000000ull;
    }
    if (!store) return;
    const double zero = __longlong_as_double(eb == kNanExp ? 0x7FF8000000000000ll : 0ll);
    const unsigned long long flip = 1ull << 63;
    auto put = [&](int m, int cp, unsigned long long b) {
      d[(long long)m * ms + cp] = __longlong_as_double((long long)b);
    };
#pragma unroll
    for (int j = 0; j < kOut; ++j) {
      if (j >= cnt) break;
      const int r = dft_r(w.p, w.row0 + n0 + j);
      const bool self = r == 0 || 2 * r == nr;
      unsigned long long b = y[j];
      put(r, cmp, b);
      // the parts that no row computes: Im at r = 0, and with s = 1 Re at n / 2
      if (r == 0) d[1] = zero;
      if (w.d.s && w.p == 2 && 2 * r == nr) d[(long long)r * ms] = zero;
      for (int m0 = nr; m0 - r <= w.d.mtop; m0 += nr) {            // a n - r and a n + r
        if (w.d.s) b ^= flip;
        if (!self) put(m0 - r, cmp, cmp ? b ^ flip : b);
        if (m0 + r <= w.d.mtop) {
          put(m0 + r, cmp, b);
          if (r == 0) d[(long long)m0 * ms + 1] = zero;
          if (w.d.s && w.p == 2 && 2 * r == nr) d[(long long)(m0 + r) * ms] = zero;
        }
      }
    }
  } else {
    // phases: e, o, se, so (cos even, cos odd, sin even, sin odd sums at sample j); the four
    // mirrored samples hold them until so is there:
    //   x_j = P - T, x_{-j} = P + T, x_{pi-j} = M + V, x_{pi+j} = M - V
    //   P, M = e +- o, T = se + so, V = se - so
    // (on the axis x_{-0} is x_0, and both sin sums are zero)
    const int nr = 4 * w.d.q, j0 = w.row0 + c;
    if (!store || (ph >= 2 && w.d.s == 0 && j0 == 0)) return;
    const bool equator = w.m == a.nnorth - 1;
    double* x = a.out[0] + (long long)(w.g * kGroupMaps) * a.map_stride;
    const long long on = ring_start(a.nside, w.m), os = ring_start(a.nside, a.nring - 1 - w.m);
    const int i1 = nr - w.d.s - j0, i2 = nr / 2 - w.d.s - j0, i3 = nr / 2 + j0;
    auto base = [&](int j) {
      return x + (long long)((n0 + j) >> 1) * a.map_stride + (((n0 + j) & 1) ? os : on);
    };
    auto live = [&](int j) { return j < cnt && !(equator && ((n0 + j) & 1)); };
    double p[kOut], q[kOut];
#pragma unroll
    for (int j = 0; j < kOut; ++j) {
      v[j] = ph >= 1 && live(j) ? base(j)[j0] : 0.0;
      p[j] = ph == 3 && live(j) ? base(j)[i2] : 0.0;
      q[j] = ph == 3 && live(j) ? base(j)[i1] : 0.0;
    }
    auto bits = [](double t) { return __double_as_longlong(t); };
    auto keep = [](long long t) { return __longlong_as_double(t); };
#pragma unroll
    for (int j = 0; j < kOut; ++j) {
      if (!live(j)) continue;
      const int ec = (int)fac[j];
      double* b = base(j);
      if (ph == 0) {
        b[j0] = keep(sum[j]);
      } else if (ph == 1) {
        b[j0] = keep(bits(v[j]) + sum[j]);
        b[i2] = keep(bits(v[j]) - sum[j]);
        if (w.d.s == 0 && j0 == 0) {                       // no later phase
          b[j0] = ec == kNanExp ? keep(0x7FF8000000000000ll)
                                : i64_scaled_any(bits(v[j]) + sum[j], ec + e);
          b[i2] = ec == kNanExp ? keep(0x7FF8000000000000ll)
                                : i64_scaled_any(bits(v[j]) - sum[j], ec + e);
        }
      } else if (ph == 2) {
        b[i1] = keep(sum[j]);
      } else {
        const long long T = bits(q[j]) + sum[j], V = bits(q[j]) - sum[j];
        const long long P = bits(v[j]), M = bits(p[j]);
        auto out = [&](long long t) {
          return ec == kNanExp ? keep(0x7FF8000000000000ll) : i64_scaled_any(t, ec + e);
        };
        b[j0] = out(P - T);
        b[i1] = out(P + T);
        b[i2] = out(M + V);
        b[i3] = out(M - V);
      }
    }
  }
}

template <int DIR, int SPIN>
__global__ void __launch_bounds__(kTcThreads, 1) k_tc_gemm(TcGemmArgs a) {
  constexpr int NPH = DIR == 0 || DIR == 2 ? 1 : DIR == 1 ? 2 : 4, NSEG = SPIN == 2 ? 2 : 1;
  constexpr bool SWAP = DIR == 3;      // matrix rows on the TMEM lanes, map columns as N
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ TcSmemHdr h;
  __shared__ UnitQueue uq;
  // per epilogue warp: its rows' factors (DIR 0), its columns' exponents (DIR 3)
  __shared__ double s_fac[kTcEpiWarps][kTcAcc];

  const int tid = threadIdx.x;
  const int warp = tc::warp_index();
  volatile int* abort = &h.abort;
  if (tid == 0) {
    for (int s = 0; s < kTcStages; ++s) {
      tc::mbar_init(&h.full[s], 1);
      tc::mbar_init(&h.empty[s], 2);                     // both UMMA warps
    }
    for (int s = 0; s < 2; ++s) {
      tc::mbar_init(&h.tfull[s], 1);
      tc::mbar_init(&h.tempty[s], kTcEpiWarps);
    }
    tc::mbar_init(&h.fin, 2);
    uq_init(uq, kTcEpiWarps + 2);
    h.abort = 0;
    tc::mbar_fence_init();
  }
  if (warp == 0) tc::tmem_alloc(&h.tmem, 512);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = h.tmem;

  uint32_t n_loaded = 0;
  if (tid == kTcEpi) {
    uint32_t i = 0;
    uq_walk(uq, a.nunits, 0, abort, [&](int u) -> bool {
      const TcUnit w = tc_unit<DIR, SPIN>(a, u);
      if (w.nk == 0) return true;
      for (int s = 0; s < NPH * NSEG; ++s) {
        const unsigned char *cols, *rows;
        int sign;
        tc_segment<DIR, SPIN>(a, w, s / NSEG, s % NSEG, cols, rows, sign);
        for (int k0 = 0; k0 < w.nk; k0 += kPartK) {
          const int nk = min(w.nk - k0, kPartK);
          // pass 0: the low half (planes 0..3) of each k-step; pass 1: both halves
          for (int j = 0; j < 3 * nk; ++j, ++i) {
            const int k = k0 + (j < nk ? j : (j - nk) >> 1);
            const uint32_t half = j < nk ? 0 : (uint32_t)((j - nk) & 1);
            const uint32_t st = i % kTcStages;
            if (!tc::mbar_wait(&h.empty[st], ((i / kTcStages) & 1) ^ 1, abort)) return false;
            unsigned char* dst = smem + st * kTcStageBytes;
            tc::mbar_arrive_expect_tx(&h.full[st], kTcStageBytes);
            tc::bulk_g2s(dst, cols + (size_t)k * kStepBytes + half * kHalfBytes, kHalfBytes,
                         &h.full[st]);
            tc::bulk_g2s(dst + kHalfBytes, rows + (size_t)k * kStepBytes + half * kHalfBytes,
                         kHalfBytes, &h.full[st]);
            ++n_loaded;
          }
        }
      }
      return true;
    });
  } else if (warp > kTcEpiWarps) {
    // UMMA warps: warp `side` issues the products of the slot pair {2 side, 2 side + 1}
    const int side = warp - kTcEpiWarps - 1;
    const uint32_t s_u = (uint32_t)tc::uniform((int)tc::smem_u32(smem));
    const uint32_t slot = (uint32_t)tc::uniform((int)tmem) + 2 * side * kCols;
    uint32_t i = 0, use = 0;       // stages consumed, passes issued (one use of every slot each)
    bool ok = true;
    auto drained = [&]() {         // the pair's sums of the pass before are out
      if (use > 0 && !tc::mbar_wait_warp(&h.tempty[side], (use - 1) & 1, abort)) return false;
      tc::tc_fence_after();
      return true;
    };
    for (uint32_t n = 0; ok; ++n) {
      const int u = uq_take(uq, n, abort);
      if (u < 0) break;
      const TcUnit w = tc_unit<DIR, SPIN>(a, u);
      // (the shuffles tell the compiler that these are warp-uniform)
      const int unk = tc::uniform(w.nk), N = tc::uniform(w.N);
      const uint32_t id1 = tc::umma_idesc_bf16(kRows, N);
      const bool wide = N > kWideN;
      for (int s = 0; s < NPH * NSEG && ok; ++s) {
        for (int k0 = 0; k0 < unk && ok; k0 += kPartK) {
          const int nk = min(unk - k0, kPartK);
          for (int k = 0; k < nk && ok; ++k, ++i) {              // pass 0
            const uint32_t st = i % kTcStages;
            if (!tc::mbar_wait_warp(&h.full[st], (i / kTcStages) & 1, abort) ||
                (k == 0 && !drained())) {
              ok = false;
              break;
            }
            tc::tc_fence_after();
            const uint64_t c0 = tc::umma_desc(s_u + st * kTcStageBytes, 128, 256);
            auto plane = [&](int d, bool second) {
              return tc::umma_desc_add(c0, (uint32_t)d * kPlaneBytes +
                                               (second != SWAP ? kHalfBytes : 0));
            };
            if (side == 0) {
              tc_products<0>(slot, plane, id1, wide, k > 0);
            } else {
              tc_products<2>(slot, plane, id1, wide, k > 0);
            }
            if (k == nk - 1) tc::umma_commit_warp(&h.tfull[side]);
            tc::umma_commit_warp(&h.empty[st]);
          }
          ++use;
          for (int k = 0; k < nk && ok; ++k, i += 2) {           // pass 1
            const uint32_t st = i % kTcStages, st1 = (i + 1) % kTcStages;
            if (!tc::mbar_wait_warp(&h.full[st], (i / kTcStages) & 1, abort) ||
                !tc::mbar_wait_warp(&h.full[st1], ((i + 1) / kTcStages) & 1, abort) ||
                (k == 0 && !drained())) {
              ok = false;
              break;
            }
            tc::tc_fence_after();
            const uint64_t ca = tc::umma_desc(s_u + st * kTcStageBytes, 128, 256);
            const uint64_t cb = tc::umma_desc(s_u + st1 * kTcStageBytes, 128, 256);
            // plane d of the UMMA's first (M) operand and of its second
            auto plane = [&](int d, bool second) {
              return tc::umma_desc_add(d < 4 ? ca : cb, (uint32_t)(d & 3) * kPlaneBytes +
                                                            (second != SWAP ? kHalfBytes : 0));
            };
            if (side == 0) {
              tc_products<4>(slot, plane, id1, wide, k > 0);
            } else {
              tc_products<6>(slot, plane, id1, wide, k > 0);
            }
            if (k == nk - 1) tc::umma_commit_warp(&h.tfull[side]);
            tc::umma_commit_warp(&h.empty[st]);
            tc::umma_commit_warp(&h.empty[st1]);
          }
          ++use;
        }
      }
    }
  } else if (tid < kTcEpi) {
    // epilogue: each warp works alone (no barrier among them); after an expired wait the
    // remaining slots are walked without work
    const int lane = tid & 31;
    const int c = ((warp & 3) << 5) + lane;              // tile column: 2 map + comp
    const int comp = c & 1;
    const int rbeg = (warp >> 2) * kTcAcc;               // this warp's quarter of the columns
    const uint32_t tbase = tmem + ((uint32_t)((warp & 3) << 5) << 16) + rbeg;
    uint32_t use = 0;
    for (uint32_t n = 0;; ++n) {
      const int u = uq_take(uq, n, abort);
      if (u < 0) break;
      const TcUnit w = tc_unit<DIR, SPIN>(a, u);
      if (w.nk == 0) continue;
      const int map = w.g * kGroupMaps + (c >> 1);
      const int ncol = 2 * min(kGroupMaps, a.kc - w.g * kGroupMaps);
      const int nrow = min(kTcAcc, (SWAP ? ncol : w.nrows) - rbeg);   // TMEM columns of this warp
      if (DIR == 0) {
        __syncwarp();
        {
          const int l = w.row0 + 2 * (rbeg + lane);
          s_fac[warp][lane] =
              l <= a.lmax ? a.tab[tri_off(w.m, a.lmax) + (l - w.m)].dm * a.pa : 0.0;
        }
        __syncwarp();
      }
      bool store = map < a.kc;
      if (DIR < 2) {
        const int4 fl = *reinterpret_cast<const int4*>(a.flags +
                                                       ((long long)w.m * a.ngroups + w.g) * 4);
        store = (fl.x | fl.y | fl.z | fl.w) == 0 && map < a.kc &&
                (DIR == 1 || !(comp == 1 && w.m == 0));
      }
      if (DIR == 3) {
        __syncwarp();
        s_fac[warp][lane] = a.EB[((long long)w.qi * a.ngroups + w.g) * kCols + rbeg + lane];
        __syncwarp();
        store = c < w.nrows;                               // the lane's matrix row
      }
#pragma unroll 1
      for (int ph = 0; ph < NPH; ++ph) {
        const int par = DIR == 0 ? w.p : ph;
        const int eb =
            DIR == 3 ? 0
                     : a.EB[((DIR == 2 ? (long long)w.qi : (long long)w.qi * 2 + par) * a.ngroups +
                             w.g) * kCols + c];
        unsigned long long acc[kTcAcc], bias = 0;
#pragma unroll
        for (int j = 0; j < kTcAcc; ++j) acc[j] = 0;
#pragma unroll 1
        for (int sg = 0; sg < NSEG; ++sg) {
          int sign = 1;
          if (SPIN == 2) {
            const unsigned char *x, *y;
            tc_segment<DIR, SPIN>(a, w, ph, sg, x, y, sign);
          }
#pragma unroll 1
          for (int k0 = 0; k0 < w.nk; k0 += kPartK) {
            const float sf = (float)sign;
            // wait for a pair of slots, drain it, hand it back
            auto pair = [&](auto P) {
              constexpr int kP = decltype(P)::value, kS = (2 * kP) & 3;
              if (!tc::mbar_wait_warp(&h.tfull[kP & 1], use & 1, abort)) return;
              tc::tc_fence_after();
              tc_drain<kP>(tbase + kS * kCols, tbase + (kS + 1) * kCols, nrow, sf, a.unit_bits,
                           acc);
              tc::tc_fence_before();
              __syncwarp();
              if (lane == 0) tc::mbar_arrive(&h.tempty[kP & 1]);
            };
            pair(std::integral_constant<int, 0>{});
            pair(std::integral_constant<int, 1>{});
            ++use;
            pair(std::integral_constant<int, 2>{});
            pair(std::integral_constant<int, 3>{});
            ++use;
            const int b = a.unit_bits;
            bias += ((unsigned long long)kBias2 << (b - 8)) +
                    ((unsigned long long)kBias2 << (b - 24)) +
                    ((unsigned long long)kBias2 << (b - 40)) + kMagic;
          }
        }
        // the phase's sums out, a few at a time: the output code exists once and the registers
        // move down to it (unrolled over all sums it ran at the instruction fetch rate, one value
        // at a time at the latency of a load)
        // (an empty column's sums are zero: any exponent does)
        const int e = (eb == kEmptyExp ? 0 : eb) - 12 - a.unit_bits +
                      (DIR == 0 ? a.eag : DIR >= 2 ? 1 : 0);
        constexpr int kOut = 4;
#pragma unroll 1
        for (int c0 = 0; c0 < nrow; c0 += kOut) {
          long long sum[kOut];
#pragma unroll
          for (int j = 0; j < kOut; ++j) sum[j] = (long long)(acc[j] - bias);
#pragma unroll
          for (int j = 0; j + kOut < kTcAcc; ++j) acc[j] = acc[j + kOut];
          tc_out<DIR, SPIN, kOut>(a, w, ph, store, c, rbeg + c0, min(kOut, nrow - c0), map, eb, e,
                                  sum, &s_fac[warp][c0]);
        }
      }
    }
  }
  // the UMMA issuer waits for its last products before TMEM is released, the loader for its
  // last copies
  if (warp > kTcEpiWarps) {
    tc::umma_commit_warp(&h.fin);
    for (uint32_t it = 0; it < tc::kWaitLimit; ++it)
      if (tc::mbar_try_wait(&h.fin, 0)) break;
  }
  if (tid == kTcEpi) {
    for (uint32_t d = 0; d < (uint32_t)kTcStages && d < n_loaded; ++d) {
      const uint32_t i = n_loaded - 1 - d;
      for (uint32_t it = 0; it < tc::kWaitLimit; ++it)
        if (tc::mbar_try_wait(&h.full[i % kTcStages], (i / kTcStages) & 1)) break;
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, 512);
  if (tid == 0 && h.abort) atomicOr(a.err, tc::kErrTimeout);
}

// ------------------------------------------------------------------ host side
size_t tc_row_bytes(const fsht_plan* p) {
  const size_t nks = (size_t)(p->nnorth + kKStep - 1) / kKStep;
  const size_t nkl = (size_t)(p->lmax / 2 + 1 + kKStep - 1) / kKStep;
  return std::max(nks, nkl) * kStepBytes;
}
int tc_groups(int kc) { return (kc + kGroupMaps - 1) / kGroupMaps; }

template <int DIR, int SPIN>
int launch_tc_gemm(const TcGemmArgs& a, cudaStream_t s) {
  FSHT_TRY(fsht_smem_limit((const void*)k_tc_gemm<DIR, SPIN>, kTcSmem));
  if (a.nunits > 0) k_tc_gemm<DIR, SPIN><<<a.nunits, kTcThreads, kTcSmem, s>>>(a);
  FSHT_LAUNCH_CHECK();
  return FSHT_OK;
}
}  // namespace

bool fsht_tc_supported(const fsht_plan* p) {
  return fsht_tc_sizes(p->nside, p->lmax);
}

int fsht_tc_tables_init(fsht_plan* p) {
  const size_t ntab = (size_t)tri_off(p->lmax + 1, p->lmax);
  FSHT_CUDA_TRY(fsht_plan_malloc(p, &p->d_lamtab, sizeof(FshtLamRow) * ntab));
  if (p->pol) {
    FSHT_CUDA_TRY(fsht_plan_malloc(p, &p->d_lamtab2, sizeof(FshtLamRow) * ntab));
    FSHT_CUDA_TRY(fsht_plan_malloc(p, &p->d_poltab, sizeof(FshtPolRow) * ntab));
  }
  k_tc_table<<<p->lmax + 1, kTabThreads, 0, p->stream>>>(p->lmax, p->d_lamtab, p->d_lamtab2,
                                                         p->d_poltab);
  FSHT_LAUNCH_CHECK();
  return fsht_wave_tables_init(p, kStepBytes);
}

int fsht_tc_wave_cap(fsht_plan* p, size_t cap) { return fsht_wave_tables_init(p, kStepBytes, cap); }

// Digit tiles of one wave of kc maps (nf = 2: Q and U or E and B, plain and i v), its exponents,
// and the flags of every order.
size_t fsht_tc_ws_bytes(const fsht_plan* p, int kc, int nf) {
  return (size_t)p->wave_qmax * 2 * tc_groups(kc) * (nf == 2 ? 4 : 1) * tc_row_bytes(p);
}
size_t fsht_tc_eb_bytes(const fsht_plan* p, int kc) {
  return (size_t)p->wave_qmax * 2 * tc_groups(kc) * kCols * sizeof(int);
}
size_t fsht_tc_flag_bytes(const fsht_plan* p, int kc) {
  return (size_t)(p->lmax + 1) * tc_groups(kc) * 4 * sizeof(int);
}

int fsht_launch_tc_slice(fsht_plan* p, int w, const double2* W0, const double2* W1,
                         unsigned char* WS, int* EB, int kc, cudaStream_t s) {
  const int* wv = p->h_waves + kWaveInts * w;
  TcSliceArgs a;
  a.W[0] = reinterpret_cast<const double*>(W0);
  a.W[1] = reinterpret_cast<const double*>(W1);
  a.kc = kc;
  a.nnorth = p->nnorth;
  a.ngroups = tc_groups(kc);
  a.q0 = wv[0];
  a.lmax = p->lmax;
  a.row_bytes = tc_row_bytes(p);
  a.ring_i0 = p->d_ring_i0;
  a.WS = WS;
  a.EB = EB;
  a.flags = p->d_tcflag;
  const dim3 grid(wv[1] - wv[0], 4 * a.ngroups);
  if (W1)
    k_tc_slice<2><<<grid, 256, 0, s>>>(a);
  else
    k_tc_slice<1><<<grid, 128, 0, s>>>(a);
  FSHT_LAUNCH_CHECK();
  return FSHT_OK;
}

int fsht_launch_tc_slice_alm(fsht_plan* p, int w, const double* alm0, const double* alm1,
                             unsigned char* WS, int* EB, int nmaps_total, int k0, int kc,
                             cudaStream_t s) {
  const int* wv = p->h_waves + kWaveInts * w;
  TcSliceAArgs a;
  a.alm[0] = alm0;
  a.alm[1] = alm1;
  a.ld = nmaps_total;
  a.k0 = k0;
  a.kc = kc;
  a.lmax = p->lmax;
  a.ngroups = tc_groups(kc);
  a.q0 = wv[0];
  a.head = fsht_tc_units_synthesis(p->lmax).head;
  a.row_bytes = tc_row_bytes(p);
  a.tab = alm1 ? p->d_lamtab2 : p->d_lamtab;
  a.WS = WS;
  a.EB = EB;
  a.flags = p->d_tcflag;
  const dim3 grid(wv[1] - wv[0], a.ngroups);
  const int cl = slice_cluster((long long)grid.x * grid.y * (alm1 ? 4 : 2), wv[5]);
  if (alm1) return launch_slice(k_tc_slice_alm<2>, grid, 512, cl, s, a);
  return launch_slice(k_tc_slice_alm<1>, grid, 256, cl, s, a);
}

namespace {
template <int SPIN, bool T>
int launch_tc_lambda(fsht_plan* p, int w, unsigned char* lbuf, cudaStream_t s) {
  const int* wv = p->h_waves + kWaveInts * w;
  if (wv[4] == 0) return FSHT_OK;
  TcLamArgs a;
  a.lmax = p->lmax;
  a.nnorth = p->nnorth;
  a.q0 = wv[0];
  a.eag = fsht_tc_eag(p->lmax);
  a.cth = p->d_cth;
  a.sth = p->d_sth;
  a.pref = p->d_pref;
  a.ring_i0 = p->d_ring_i0;
  a.tab = SPIN == 2 ? p->d_lamtab2 : p->d_lamtab;
  a.ptab = p->d_poltab;
  a.lam_off = T ? p->d_lam_offT : p->d_lam_off;
  a.lbuf = lbuf;
  const dim3 grid(wv[1] - wv[0], wv[4]);
  if (T)
    k_tc_lambda_T<SPIN><<<grid, 128, 0, s>>>(a);
  else
    k_tc_lambda<SPIN><<<grid, 128, 0, s>>>(a);
  FSHT_LAUNCH_CHECK();
  return FSHT_OK;
}
}  // namespace

int fsht_launch_tc_lambda(fsht_plan* p, int w, unsigned char* lbuf, cudaStream_t s) {
  return launch_tc_lambda<0, false>(p, w, lbuf, s);
}
int fsht_launch_tc_lambda_pol(fsht_plan* p, int w, unsigned char* lbuf, cudaStream_t s) {
  return launch_tc_lambda<2, false>(p, w, lbuf, s);
}
int fsht_launch_tc_lambdaT(fsht_plan* p, int w, unsigned char* lbuf, cudaStream_t s) {
  return launch_tc_lambda<0, true>(p, w, lbuf, s);
}
int fsht_launch_tc_lambdaT_pol(fsht_plan* p, int w, unsigned char* lbuf, cudaStream_t s) {
  return launch_tc_lambda<2, true>(p, w, lbuf, s);
}

int fsht_launch_tc_gemm(fsht_plan* p, int w, int dir, int spin, const unsigned char* WS,
                        const int* EB, const unsigned char* lbuf, double* out0, double* out1,
                        int nmaps_total, int k0, int kc, int accumulate, int which,
                        cudaStream_t s) {
  const int* wv = p->h_waves + kWaveInts * w;
  TcGemmArgs a;
  a.lmax = p->lmax;
  a.nnorth = p->nnorth;
  a.ngroups = tc_groups(kc);
  a.q0 = wv[0];
  a.q1 = wv[1];
  a.ntmax = dir == 0 ? wv[2] : wv[4];
  a.nfield = 1;
  a.field0 = 0;
  if (spin == 2) {
    a.nfield = which == 3 ? 2 : 1;
    a.field0 = which == 2 ? 1 : 0;
  }
  a.accumulate = accumulate;
  a.unit_bits = (dir == 0 ? fsht_tc_units_analysis(p->nside, p->lmax)
                          : fsht_tc_units_synthesis(p->lmax)).bits;
  a.eag = fsht_tc_eag(p->lmax);
  a.row_bytes = tc_row_bytes(p);
  a.ring_i0 = p->d_ring_i0;
  a.lam_off = dir == 0 ? p->d_lam_off : p->d_lam_offT;
  a.tab = spin == 2 ? p->d_lamtab2 : p->d_lamtab;
  a.lbuf = lbuf;
  a.WS = WS;
  a.EB = EB;
  a.flags = p->d_tcflag;
  a.out[0] = out0;
  a.out[1] = out1;
  a.ld = nmaps_total;
  a.k0 = k0;
  a.kc = kc;
  a.pa = spin == 0 ? p->pa : -p->pa;
  a.err = p->d_err;
  a.nunits = a.ngroups * a.nfield * (dir == 0 ? 2 : 1) * a.ntmax * (wv[1] - wv[0]);
  if (dir == 0)
    return spin == 0 ? launch_tc_gemm<0, 0>(a, s) : launch_tc_gemm<0, 2>(a, s);
  return spin == 0 ? launch_tc_gemm<1, 0>(a, s) : launch_tc_gemm<1, 2>(a, s);
}

// ------------------------------------------------------------------ ring transforms, host side
namespace {
// The belt takes the matrix form up to this nside: its products grow with nside^3 in all, the
// power-of-two FFT's passes with nside^2 log nside.
constexpr int kDftBeltMax = 256;

// Units of the forward (two rings added: 1) and inverse transforms (four samples: 2) of a plan.
FshtTcUnits dft_units(const fsht_plan* p, int extra) {
  return fsht_tc_units_dft(p->nside <= kDftBeltMax ? p->nside + 1 : p->nside - 1, extra);
}

DftSliceArgs dft_slice_args(const fsht_plan* p, const int* wv, int ngroups, int extra) {
  DftSliceArgs a{};
  a.rings = p->d_dft + wv[0];
  a.ngroups = ngroups;
  a.head = dft_units(p, extra).head;
  a.WS = p->d_ws;
  a.EB = p->d_eb;
  a.nside = p->nside;
  a.nring = p->nring;
  a.nnorth = p->nnorth;
  return a;
}

template <bool INV>
int launch_dft_trig(fsht_plan* p, const int* wv, cudaStream_t s) {
  DftTrigArgs a;
  a.rings = p->d_dft + wv[0];
  a.cosv = p->d_dft_cos;
  a.lbuf = p->d_lbuf;
  const size_t sm = sizeof(long long) * (2 * (size_t)wv[3] + 1);
  FSHT_TRY(fsht_smem_limit((const void*)k_dft_trig<INV>, sm));
  k_dft_trig<INV><<<dim3(wv[1] - wv[0], 4 * wv[2]), 256, sm, s>>>(a);
  FSHT_LAUNCH_CHECK();
  return FSHT_OK;
}

TcGemmArgs dft_gemm_args(const fsht_plan* p, const int* wv, int ngroups, int cnt, int extra) {
  TcGemmArgs a{};
  a.ngroups = ngroups;
  a.ntmax = wv[2];
  a.nnorth = p->nnorth;
  a.unit_bits = dft_units(p, extra).bits;
  a.lbuf = p->d_lbuf;
  a.WS = p->d_ws;
  a.EB = p->d_eb;
  a.kc = cnt;
  a.err = p->d_err;
  a.rings = p->d_dft + wv[0];
  a.nside = p->nside;
  a.nring = p->nring;
  return a;
}
}  // namespace

// The rings of the matrix form in waves whose matrix tiles fit the lambda staging buffer and
// whose digit tiles fit one 64-map group's share of the contraction's; belt rings of one phase
// share their matrices.
int fsht_dft_tables_init(fsht_plan* p) {
  const int ns = p->nside;
  const int end = ns <= kDftBeltMax ? 2 * ns : ns - 1;
  p->dft_end = 0;
  std::vector<FshtDftRing> rings;
  std::vector<int> order;
  for (int i = ns - 2; i >= 0; --i) order.push_back(i);            // caps, large first
  if (end > ns)
    for (int s = 1; s >= 0; --s)
      for (int i = ns - 1; i < 2 * ns; ++i)
        if (ring_phase_flag(ns, i) == s) order.push_back(i);
  // the staging buffer holds at least the largest ring's matrices, and all of a small plan's
  const long long unit = kStepBytes;
  const long long nkm = (ns + 16) / 16, nrm = (ns + 128) / 128;
  const long long want =
      std::max<long long>(4 * nkm * nrm, std::min<long long>(2048, 2LL * ns * ns / 16));
  p->lbuf_bytes = std::max<size_t>(p->lbuf_bytes, (size_t)(want * unit));
  const long long cap_t = (long long)(p->lbuf_bytes / unit);
  const long long cap_c = (long long)(fsht_tc_ws_bytes(p, 1, 1) / unit);
  const int cap_r = 2 * p->wave_qmax;
  std::vector<int> waves;
  long long ut = 0, uc = 0, ucos = 0;
  int w0 = 0, nrt = 0, qm = 0, tiles = 0;
  std::vector<long long> cls(2, -1), clsc(2, -1);                  // belt classes of this wave
  auto close = [&](int e) {
    if (e > w0) {
      const int wv[kDftWaveInts] = {w0, e, nrt, qm, (int)uc, tiles};
      waves.insert(waves.end(), wv, wv + kDftWaveInts);
    }
    w0 = e;
    ut = uc = 0;
    nrt = qm = tiles = 0;
    cls[0] = cls[1] = -1;
  };
  for (int i : order) {
    FshtDftRing d{};
    d.ring = i;
    d.q = std::min(i + 1, ns);
    d.s = ring_phase_flag(ns, i);
    d.nk = (d.q + (d.s == 0) + kKStep - 1) / kKStep;
    d.nrt = (d.q + (d.s == 0) + kRows - 1) / kRows;
    d.mtop = -1;
    for (int m = p->lmax; m >= 0; --m)
      if (p->h_ring_i0[m] <= i) {
        d.mtop = m;
        break;
      }
    const bool belt = d.q == ns;
    const long long tsteps = 4LL * d.nrt * d.nk, csteps = 4LL * d.nk;
    if (tsteps > cap_t || csteps > cap_c) return FSHT_OK;          // no matrix form
    bool fresh = !belt || cls[d.s] < 0;
    if (ut + (fresh ? tsteps : 0) > cap_t || uc + csteps > cap_c ||
        (int)rings.size() - w0 >= cap_r) {
      close((int)rings.size());
      fresh = true;
    }
    d.first = fresh ? 1 : 0;
    if (fresh) {
      d.off_t = ut;
      ut += tsteps;
      if (belt) cls[d.s] = d.off_t;
    } else {
      d.off_t = cls[d.s];
    }
    if (belt && clsc[d.s] >= 0) {
      d.off_cos = clsc[d.s];
    } else {
      d.off_cos = ucos;
      ucos += 2LL * d.q + 1;
      if (belt) clsc[d.s] = d.off_cos;
    }
    d.off_c = uc;
    uc += csteps;
    nrt = std::max(nrt, d.nrt);
    tiles += d.nrt;
    qm = std::max(qm, d.q);
    rings.push_back(d);
  }
  close((int)rings.size());
  if (rings.empty()) return FSHT_OK;
  p->ndft_waves = (int)waves.size() / kDftWaveInts;
  p->h_dft_waves = new (std::nothrow) int[waves.size()];
  if (!p->h_dft_waves) {
    fsht_set_error("host allocation failed");
    return FSHT_ENOMEM;
  }
  std::copy(waves.begin(), waves.end(), p->h_dft_waves);
  FSHT_CUDA_TRY(fsht_plan_malloc(p, &p->d_dft, sizeof(FshtDftRing) * rings.size()));
  FSHT_CUDA_TRY(fsht_plan_malloc(p, &p->d_dft_cos, sizeof(long long) * ucos));
  FSHT_CUDA_TRY(cudaMemcpyAsync(p->d_dft, rings.data(), sizeof(FshtDftRing) * rings.size(),
                                cudaMemcpyHostToDevice, p->stream));
  k_dft_cos<<<(unsigned)rings.size(), 256, 0, p->stream>>>(p->d_dft, p->d_dft_cos);
  FSHT_LAUNCH_CHECK();
  FSHT_CUDA_TRY(cudaStreamSynchronize(p->stream));                 // the list is a local vector
  p->dft_end = end;
  return FSHT_OK;
}

// Maps [k0, k0 + cnt) of a chunk of kc maps (maps: the chunk's base; host: in host memory, read in
// place) -> their {S, D} of rings below dft_end.
int fsht_launch_dft_fwd(fsht_plan* p, const double* maps, long long map_stride, int kc, int k0,
                        int cnt, bool host, double2* W, cudaStream_t s) {
  const int ngroups = tc_groups(cnt);
  for (int w = 0; w < p->ndft_waves; ++w) {
    const int* wv = p->h_dft_waves + kDftWaveInts * w;
    FSHT_TRY(launch_dft_trig<false>(p, wv, s));
    DftSliceArgs sa = dft_slice_args(p, wv, ngroups, 1);
    sa.maps = maps + (long long)k0 * map_stride;
    sa.map_stride = map_stride;
    sa.cnt = cnt;
    if (host) {
      const size_t sm = sizeof(double) * 8 * (size_t)wv[3];        // two rings of 4 q samples
      FSHT_TRY(fsht_smem_limit((const void*)k_dft_slice<1>, sm));
      k_dft_slice<1><<<dim3(wv[1] - wv[0], cnt), 256, sm, s>>>(sa);
    } else {
      k_dft_slice<4><<<dim3(wv[1] - wv[0], (cnt + 3) / 4), 256, 0, s>>>(sa);
    }
    FSHT_LAUNCH_CHECK();
    TcGemmArgs a = dft_gemm_args(p, wv, ngroups, cnt, 1);
    a.k_off = k0;
    a.w_kc = kc;
    a.out[0] = reinterpret_cast<double*>(W);
    a.nunits = ngroups * 4 * a.ntmax * (wv[1] - wv[0]);
    FSHT_TRY((launch_tc_gemm<2, 0>(a, s)));
  }
  return FSHT_OK;
}

// {G_N, G_S} of rings below dft_end -> their pixels, the first cnt of kc maps.
int fsht_launch_dft_inv(fsht_plan* p, const double2* W, double* maps, long long map_stride, int kc,
                        int cnt, cudaStream_t s) {
  const int ngroups = tc_groups(cnt);
  for (int w = 0; w < p->ndft_waves; ++w) {
    const int* wv = p->h_dft_waves + kDftWaveInts * w;
    FSHT_TRY(launch_dft_trig<true>(p, wv, s));
    DftSliceArgs sa = dft_slice_args(p, wv, ngroups, 2);
    sa.W = W;
    sa.kc = kc;
    sa.cnt = cnt;
    k_dft_slice_inv<<<dim3(wv[1] - wv[0], (cnt + 15) / 16), 256, 0, s>>>(sa);
    FSHT_LAUNCH_CHECK();
    TcGemmArgs a = dft_gemm_args(p, wv, ngroups, cnt, 2);
    a.map_stride = map_stride;
    a.out[0] = maps;
    a.nunits = ngroups * a.ntmax * (wv[1] - wv[0]);
    FSHT_TRY((launch_tc_gemm<3, 0>(a, s)));
  }
  return FSHT_OK;
}
