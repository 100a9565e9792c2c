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
// FP32 rounding is far below FP64's.  The epilogue adds every level into one 64-bit integer per output element
// (unit 2^-unit_bits), so no FP64 instruction runs before the last conversion and the order of
// the parts does not matter.
//
// What the fixed point costs: the dropped levels (8 and up) and the unit are below 2^-44 of
// the largest operand pair.  Against long-double sums (white, smooth and constant columns,
// nside 64..1024) the error is 0.2..1 times that of an FP64 FMA loop for white and constant
// columns.  Columns that the fixed point cannot hold (non-finite, or a maximum beyond 2^+-900)
// are flagged per (order, 64-map group) and contracted by the FMA kernels (legendre_fp64.cu).
//
// Per wave of orders:
//   k_tc_slice      {S, D} phases -> digit tiles and column exponents       (HBM bound)
//   k_tc_lambda     FP64 recursion -> lambda digit tiles, once for all maps (FP64 pipe)
//   k_tc_gemm       persistent tcgen05 contraction                          (tensor pipe)
// and for the synthesis k_tc_slice_alm, k_tc_lambda_T and k_tc_gemm<1, *>.
#include "legendre_rec.cuh"
#include "split_common.cuh"

#include <algorithm>
#include <cmath>

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
// operations per clock per SM.  |v 2^k| < 2^62 is the caller's scale.
__device__ __forceinline__ unsigned long long fixed_biased(double v, int k) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  const int ex = (int)(b >> 52) & 0x7FF;
  const unsigned long long mant = (b & 0xFFFFFFFFFFFFFull) | (1ull << 52);
  const int sh = ex - 1075 + k;
  unsigned long long x = 0;
  if (ex != 0 && sh > -53) x = sh >= 0 ? mant << min(sh, 9) : mant >> -sh;
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

// a 2^e as the nearest FP64, with integer instructions; zero below the normal range.
__device__ __forceinline__ double i64_scaled(long long a, int e) {
  unsigned long long u = (unsigned long long)(a < 0 ? -a : a);
  if (u == 0) return 0.0;
  const int lz = __clzll((long long)u);
  u <<= lz;
  const unsigned long long r = (u >> 11) + ((u >> 10) & 1);       // 2^52 .. 2^53
  const int ex = 63 - lz + e + 1023;
  if (ex <= 0) return 0.0;
  unsigned long long b = ((unsigned long long)ex << 52) + (r - (1ull << 52));
  b |= a < 0 ? 1ull << 63 : 0ull;
  return __longlong_as_double((long long)b);
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
    r.dm = 1.0;
    r.dx = 0;
    r.erow = ilogb(bound) + 1;
    tab2[base + j] = r;
    FshtPolRow c{0.0, 0.0, 0.0, 0.0};
    if (j > 0) {
      const RecConst rc = rec_coeffs((int)L, m);
      c.c1 = rc.a;
      c.c2 = rc.b;
    }
    c.c3 = lam_fact((int)L, m);
    c.c4 = normal_l((int)L);
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
// it, plus Dx for spin 0).
template <int SPIN>
__device__ __forceinline__ void tc_value(TcRing& r, int j, int m, double beta, const FshtPolRow& c,
                                         int k, unsigned long long& y1, unsigned long long& y2) {
  if (SPIN == 2) {
    if (j > 0) rec_step(r.s1, r.s2, r.et, c.c1 * r.x, c.c2);
    y1 = y2 = kBias;
    if (r.et != 0) return;
    double l1, l2;
    pol_lambda(r.pol, m + j, m, r.s1, r.s2, c.c3, c.c4, l1, l2);
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
      if (SPIN == 2) s_c[tid] = ptab[lb + tid];
    }
    __syncthreads();
    if (SPIN == 0) tc_rescale(R);
#pragma unroll 4
    for (int jj = 0; jj < LB; ++jj) {
      const int j = lb + jj;
      unsigned long long y1 = kBias, y2 = kBias;
      if (j < nl && valid)
        tc_value<SPIN>(R, j, m, s_beta[jj], s_c[SPIN == 2 ? jj : 0], s_k[jj], y1, y2);
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
      if (SPIN == 2) s_c[tid] = ptab[lb + tid];
    }
    __syncthreads();
    if (SPIN == 0) tc_rescale(R);
    unsigned long long y[NT][2][8];
#pragma unroll
    for (int jj = 0; jj < LB; ++jj) {
      const int j = lb + jj;
      unsigned long long y1 = kBias, y2 = kBias;
      if (j < nl && valid)
        tc_value<SPIN>(R, j, m, s_beta[jj], s_c[SPIN == 2 ? jj : 0], s_k[jj], y1, y2);
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
// grid (q in wave, group), 128 threads per field = (comp, map): v = a_lm Dm 2^EA(l), tile column
// c = 2 map + comp, 16 l of one parity per k-step.  T: an exponent per (column, parity), since
// the two parities are separate sums; E/B (NF = 2): one per map and order, plain and i v copies.
struct TcSliceAArgs {
  const double* alm[2];
  int ld, k0, kc, lmax, ngroups, q0;
  size_t row_bytes;
  const FshtLamRow* tab;
  unsigned char* WS;
  int* EB;
  int* flags;
};

template <int NF>
__global__ void __launch_bounds__(128 * NF) k_tc_slice_alm(TcSliceAArgs a) {
  __shared__ unsigned long long s_mx[2 * NF][64];
  const int qi = blockIdx.x, g = blockIdx.y;
  const int m = m_of_q(a.q0 + qi, a.lmax);
  const int f = NF == 1 ? 0 : (int)(threadIdx.x >> 7);
  const int kl = threadIdx.x & 63, comp = (threadIdx.x >> 6) & 1;
  const int k = g * kGroupMaps + kl;
  const int c = 2 * kl + comp;
  const bool valid = k < a.kc && !(comp == 1 && m == 0);
  const long long L1 = a.lmax + 1;
  const int nkl = ((a.lmax - m) / 2 + 1 + kKStep - 1) / kKStep;
  const FshtLamRow* tab = a.tab + tri_off(m, a.lmax);
  const double* col = a.alm[f] + a.k0 + k +
                      (comp == 0 ? (long long)m * L1 + m : (L1 - m) * L1) * a.ld;
  auto cnt_of = [&](int p) { return a.lmax - m - p >= 0 ? (a.lmax - m - p) / 2 + 1 : 0; };
  // bits of |a Dm| 2^EA(l); values too small for the exponent sum count as zero (the flag of a
  // tiny column maximum sends the whole column to the FMA kernel)
  auto key_of = [&](double w, int ea) -> unsigned long long {
    const unsigned long long b =
        (unsigned long long)__double_as_longlong(w) & 0x7FFFFFFFFFFFFFFFull;
    if ((b >> 52) < 32) return b ? 1ull : 0ull;
    if ((b >> 52) > 2000) return 0x7FF0000000000000ull;
    return b + ((unsigned long long)(long long)ea << 52);
  };
  bool flag = false;
  unsigned long long mxp[2];
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    unsigned long long mx = 0;
    if (valid) {
      const int cnt = cnt_of(p);
#pragma unroll 8
      for (int idx = 0; idx < cnt; ++idx) {
        const int j = p + 2 * idx;
        const FshtLamRow rw = tab[j];
        mx = max(mx, key_of(col[(long long)j * a.ld] * rw.dm, rw.erow + rw.dx));
      }
    }
    mxp[p] = mx;
  }
  if (NF == 2) {
    __syncthreads();
    s_mx[f * 2 + comp][kl] = max(mxp[0], mxp[1]);
    __syncthreads();
    unsigned long long mx = 0;
#pragma unroll
    for (int h = 0; h < 2 * NF; ++h) mx = max(mx, s_mx[h][kl]);
    mxp[0] = mxp[1] = mx;
  }
  int Ep[2];
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    const int ef = (int)(mxp[p] >> 52);
    const bool odd_range = mxp[p] != 0 && (ef < 1023 - kMaxExp || ef > 1023 + kMaxExp);
    flag |= odd_range;
    Ep[p] = (mxp[p] == 0 || odd_range) ? kEmptyExp : ef - 1022;
    if (f == 0) a.EB[(((long long)qi * 2 + p) * a.ngroups + g) * kCols + c] = Ep[p];
  }
  const int any = __syncthreads_or(flag ? 1 : 0);
  if (threadIdx.x < 4) a.flags[((long long)m * a.ngroups + g) * 4 + threadIdx.x] = any;
  constexpr int NC = NF == 1 ? 1 : 4;
  const int cr = 2 * kl + (comp ^ 1);
#pragma unroll 1
  for (int p = 0; p < 2; ++p) {
    const int cnt = cnt_of(p), E = p ? Ep[1] : Ep[0];
    unsigned char* base =
        a.WS + (((size_t)(qi * 2 + p) * a.ngroups + g) * NC + 2 * f) * a.row_bytes;
    unsigned char* dst = base + (c >> 3) * 256 + (c & 7) * 16;
    unsigned char* rot = base + a.row_bytes + (cr >> 3) * 256 + (cr & 7) * 16;
    for (int h = 0; h < 2 * nkl; ++h) {
      unsigned long long y[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int idx = h * 8 + j;
        y[j] = kBias;
        if (valid && idx < cnt && E != kEmptyExp) {
          const FshtLamRow rw = tab[p + 2 * idx];
          y[j] = fixed_biased(col[(long long)(p + 2 * idx) * a.ld] * rw.dm,
                              rw.erow + rw.dx + kFixBits - E);
        }
      }
      store_planes<NF == 2>(dst + (size_t)(h >> 1) * kStepBytes + (h & 1) * 128,
                            rot + (size_t)(h >> 1) * kStepBytes + (h & 1) * 128, comp == 1, y);
    }
  }
}

// ------------------------------------------------------------------ contraction
// Persistent, one CTA per SM, units from the queue of split_common.cuh.  A unit is a 128-column (64 maps x Re/Im, the UMMA M side = TMEM
// lanes) x N-row tile: N <= 128 l-rows of one parity (DIR 0, analysis) or rings (DIR 1,
// synthesis), over one or two phases of one or two segments:
//   DIR 0          one phase;  spin 2: lambda1 against the field, lambda2 against i x the other
//   DIR 1          phase 0 gives A, phase 1 gives B', north = A + B', south = A - B':
//                  T: even l, then odd l; Q/U: (lambda1 even, lambda2 odd), then (lambda1 odd,
//                  lambda2 even), since lambda1 keeps (-1)^(l-m) and lambda2 takes the opposite
// Each part of <= 12 k-steps runs two passes through the four 128-column TMEM accumulators:
// levels 0..3 (digit planes 0..3) and levels 4..7 (all planes).  A level's accumulator is drained
// into the 64-bit integers as soon as its last product is done, while the products of the other
// levels still run, and is handed back alone: the four slots have their own barriers.
// Warps 0-7: epilogue (two per TMEM lane quarter, one per half of the rows), warp 8 lane 0:
// copies (16 KB of each operand per stage), warp 9 lane 0: UMMAs.
// The map columns are on the lanes, so a warp's alm stores are two 128-byte segments and its
// phase-matrix stores whole {Re, Im} pairs, with no staging through shared memory.
constexpr int kTcThreads = kEpiThreads + 96;     // epilogue, copy thread's warp, two UMMA warps
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
};

struct __align__(8) TcSmemHdr {
  uint64_t full[kTcStages], empty[kTcStages], tfull[4], tempty[4], fin;
  uint32_t tmem;
  int abort;
};

struct TcUnit {
  int g, field, p, t, qi, m, nk, nt, row0, nrows, N;
};

template <int DIR, int SPIN>
__device__ __forceinline__ TcUnit tc_unit(const TcGemmArgs& a, int u) {
  TcUnit w;
  w.g = u % a.ngroups;
  int r = u / a.ngroups;
  w.field = 0;
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

// Segment sg of phase ph: its column tiles, lambda tiles and sign.
template <int DIR, int SPIN>
__device__ __forceinline__ void tc_segment(const TcGemmArgs& a, const TcUnit& w, int ph, int sg,
                                           const unsigned char*& cols, const unsigned char*& rows,
                                           int& sign) {
  constexpr int NT = SPIN == 2 ? 2 : 1, NC = SPIN == 2 ? 4 : 1;
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

// acc += level sums L of one slot, 64 rows per thread: f L (an integer, or rounded to one) times
// mul, in the high word (HI) or as a 32 x 32 + 64-bit multiply-add.  The integer comes out of
// the mantissa of f L + 1.5 2^23, so a sum costs a float FMA, a maximum and the multiply-add (the
// conversion instruction and its 64-bit handling took three times as long, with the UMMA warps
// waiting); the bias 0x4B400000 stays in acc until the end of the unit.  Sums of 2^22 and more,
// which need extreme digits throughout, take the conversion.
constexpr uint32_t kMagic = 0x4B400000u;
template <bool HI>
__device__ __forceinline__ void tc_drain(uint32_t taddr, int nrow, float f, uint32_t mul,
                                         unsigned long long (&acc)[64]) {
#pragma unroll
  for (int c = 0; c < 64; c += 32) {
    if (c >= nrow) break;
    uint32_t v0[16], v1[16];
    tc::tmem_ld16(taddr + c, v0);
    tc::tmem_ld16(taddr + c + 16, v1);
    tc::tmem_wait_ld();
    float mx = 0.f;
    auto L = [&](int j) { return __uint_as_float(j < 16 ? v0[j & 15] : v1[j & 15]); };
#pragma unroll
    for (int j = 0; j < 32; ++j) mx = fmaxf(mx, fabsf(L(j)));
    const bool big = __any_sync(0xffffffffu, mx * fabsf(f) >= 0x1p22f);
    auto put = [&](int j, uint32_t n) {
      if (HI)
        acc[c + j] = ((unsigned long long)((uint32_t)(acc[c + j] >> 32) + n * mul) << 32) |
                     (uint32_t)acc[c + j];
      else
        acc[c + j] += (unsigned long long)n * mul;
    };
    if (!big) {
#pragma unroll
      for (int j = 0; j < 32; ++j) put(j, __float_as_uint(fmaf(L(j), f, 12582912.f)));
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j) put(j, (uint32_t)__float2int_rn(L(j) * f) + kMagic);
    }
  }
}

template <int DIR, int SPIN>
__global__ void __launch_bounds__(kTcThreads, 1) k_tc_gemm(TcGemmArgs a) {
  constexpr int NPH = DIR == 0 ? 1 : 2, NSEG = SPIN == 2 ? 2 : 1;
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ TcSmemHdr h;
  __shared__ UnitQueue uq;
  __shared__ double s_fac[kEpiThreads / 32][64];      // per epilogue warp: its rows' factors

  const int tid = threadIdx.x;
  const int warp = tc::warp_index();
  volatile int* abort = &h.abort;
  if (tid == 0) {
    for (int s = 0; s < kTcStages; ++s) {
      tc::mbar_init(&h.full[s], 1);
      tc::mbar_init(&h.empty[s], 2);                     // both UMMA warps
    }
    for (int s = 0; s < 4; ++s) {
      tc::mbar_init(&h.tfull[s], 1);
      tc::mbar_init(&h.tempty[s], kEpiThreads / 32);
    }
    tc::mbar_init(&h.fin, 2);
    uq_init(uq, kEpiThreads / 32 + 2);
    h.abort = 0;
    tc::mbar_fence_init();
  }
  if (warp == 0) tc::tmem_alloc(&h.tmem, 512);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = h.tmem;

  uint32_t n_loaded = 0;
  if (tid == kEpiThreads) {
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
  } else if (warp > kEpiThreads / 32) {
    // UMMA warps: slots 0 and 3, and slots 1 and 2 (5 of 10 and 13 of 26 products each)
    const int side = warp - kEpiThreads / 32 - 1;
    const uint32_t s_u = (uint32_t)tc::uniform((int)tc::smem_u32(smem));
    const uint32_t utmem = (uint32_t)tc::uniform((int)tmem);
    uint32_t i = 0, use = 0;       // stages consumed, passes issued (one use of every slot each)
    bool ok = true;
    for (uint32_t n = 0; ok; ++n) {
      const int u = uq_take(uq, n, abort);
      if (u < 0) break;
      const TcUnit w = tc_unit<DIR, SPIN>(a, u);
      // (the shuffles tell the compiler that these are warp-uniform)
      const int unk = tc::uniform(w.nk);
      const uint32_t idesc = tc::umma_idesc_bf16(kRows, tc::uniform(w.N));
      for (int s = 0; s < NPH * NSEG && ok; ++s) {
        for (int k0 = 0; k0 < unk && ok; k0 += kPartK) {
          const int nk = min(unk - k0, kPartK);
          for (int k = 0; k < nk && ok; ++k, ++i) {              // pass 0
            const uint32_t st = i % kTcStages;
            if (!tc::mbar_wait_warp(&h.full[st], (i / kTcStages) & 1, abort)) {
              ok = false;
              break;
            }
            tc::tc_fence_after();
            const uint64_t ca = tc::umma_desc(s_u + st * kTcStageBytes, 128, 256);
            const uint64_t ra = tc::umma_desc_add(ca, kHalfBytes);
#pragma unroll
            for (int lev = 0; lev < 4; ++lev) {
              if ((lev == 0 || lev == 3) != (side == 0)) continue;
              if (k == 0 && use > 0) {
                if (!tc::mbar_wait_warp(&h.tempty[lev], (use - 1) & 1, abort)) {
                  ok = false;
                  break;
                }
                tc::tc_fence_after();
              }
#pragma unroll
              for (int aa = 0; aa <= lev; ++aa)
                tc::umma_bf16_warp(utmem + lev * kCols, tc::umma_desc_add(ca, aa * kPlaneBytes),
                                   tc::umma_desc_add(ra, (lev - aa) * kPlaneBytes), idesc,
                                   (k > 0 || aa > 0) ? 1u : 0u);
              if (k == nk - 1) tc::umma_commit_warp(&h.tfull[lev]);
            }
            if (ok) tc::umma_commit_warp(&h.empty[st]);
          }
          ++use;
          for (int k = 0; k < nk && ok; ++k, i += 2) {           // pass 1
            const uint32_t st = i % kTcStages, st1 = (i + 1) % kTcStages;
            if (!tc::mbar_wait_warp(&h.full[st], (i / kTcStages) & 1, abort) ||
                !tc::mbar_wait_warp(&h.full[st1], ((i + 1) / kTcStages) & 1, abort)) {
              ok = false;
              break;
            }
            tc::tc_fence_after();
            const uint64_t ca = tc::umma_desc(s_u + st * kTcStageBytes, 128, 256);
            const uint64_t cb = tc::umma_desc(s_u + st1 * kTcStageBytes, 128, 256);
            auto plane = [&](int d) {
              return tc::umma_desc_add(d < 4 ? ca : cb, (uint32_t)(d & 3) * kPlaneBytes);
            };
#pragma unroll
            for (int lev = 4; lev < 8; ++lev) {
              if ((lev == 4 || lev == 7) != (side == 0)) continue;
              if (k == 0) {
                if (!tc::mbar_wait_warp(&h.tempty[lev - 4], (use - 1) & 1, abort)) {
                  ok = false;
                  break;
                }
                tc::tc_fence_after();
              }
#pragma unroll
              for (int aa = 0; aa <= lev; ++aa)
                tc::umma_bf16_warp(utmem + (lev - 4) * kCols, plane(aa),
                                   tc::umma_desc_add(plane(lev - aa), kHalfBytes), idesc,
                                   (k > 0 || aa > 0) ? 1u : 0u);
              if (k == nk - 1) tc::umma_commit_warp(&h.tfull[lev - 4]);
            }
            if (ok) {
              tc::umma_commit_warp(&h.empty[st]);
              tc::umma_commit_warp(&h.empty[st1]);
            }
          }
          ++use;
        }
      }
    }
  } else if (tid < kEpiThreads) {
    // epilogue: each warp works alone (no barrier among them); after an expired wait the
    // remaining slots are walked without work
    const int lane = tid & 31;
    const int c = ((warp & 3) << 5) + lane;              // tile column: 2 map + comp
    const int comp = c & 1;
    const int rbeg = (warp >> 2) * 64;                   // this warp's half of the rows
    const uint32_t tbase = tmem + ((uint32_t)((warp & 3) << 5) << 16) + rbeg;
    const long long L1 = a.lmax + 1;
    // level weights 2^wt, wt = unit_bits - 8 s, as (float factor, integer multiplier): 2^32 and up
    // in the high word, the others with multipliers <= 2^30
    uint32_t use = 0;
    for (uint32_t n = 0;; ++n) {
      const int u = uq_take(uq, n, abort);
      if (u < 0) break;
      const TcUnit w = tc_unit<DIR, SPIN>(a, u);
      if (w.nk == 0) continue;
      const int map = w.g * kGroupMaps + (c >> 1);
      const int nrow = min(64, w.nrows - rbeg);
      if (DIR == 0) {
        __syncwarp();
        for (int j = lane; j < 64; j += 32) {
          const int l = w.row0 + 2 * (rbeg + j);
          s_fac[warp][j] = l <= a.lmax ? a.tab[tri_off(w.m, a.lmax) + (l - w.m)].dm * a.pa : 0.0;
        }
        __syncwarp();
      }
      const int4 fl = *reinterpret_cast<const int4*>(a.flags +
                                                     ((long long)w.m * a.ngroups + w.g) * 4);
      const bool store = (fl.x | fl.y | fl.z | fl.w) == 0 && map < a.kc &&
                         (DIR == 1 || !(comp == 1 && w.m == 0));
#pragma unroll 1
      for (int ph = 0; ph < NPH; ++ph) {
        const int par = DIR == 0 ? w.p : ph;
        const int eb = a.EB[(((long long)w.qi * 2 + par) * a.ngroups + w.g) * kCols + c];
        unsigned long long acc[64], bias = 0;
#pragma unroll
        for (int j = 0; j < 64; ++j) acc[j] = 0;
#pragma unroll 1
        for (int sg = 0; sg < NSEG; ++sg) {
          int sign = 1;
          if (SPIN == 2) {
            const unsigned char *x, *y;
            tc_segment<DIR, SPIN>(a, w, ph, sg, x, y, sign);
          }
#pragma unroll 1
          for (int k0 = 0; k0 < w.nk; k0 += kPartK) {
#pragma unroll 1
            for (int lev = 0; lev < 8; ++lev) {
              const int slot = lev & 3;
              const bool ok = tc::mbar_wait_warp(&h.tfull[slot], use & 1, abort);
              if (slot == 3) ++use;
              if (!ok) continue;
              tc::tc_fence_after();
              const int wt = a.unit_bits - 8 * lev;      // weight 2^wt of this level
              if (wt >= 32) {
                tc_drain<true>(tbase + slot * kCols, nrow, (float)sign, 1u << (wt - 32), acc);
                bias += (unsigned long long)kMagic << wt;
              } else {
                const int me = min(max(wt, 0), 30);
                tc_drain<false>(tbase + slot * kCols, nrow, sign * ldexpf(1.f, wt - me), 1u << me,
                                acc);
                bias += (unsigned long long)kMagic << me;
              }
              tc::tc_fence_before();
              tc::mbar_arrive_warp(&h.tempty[slot]);
            }
          }
        }
        // the phase's sums out
        const int e = eb - 12 - a.unit_bits + (DIR == 0 ? a.eag : 0);
        if (!store) continue;
        if (DIR == 0) {
          double* out = a.out[SPIN == 2 ? w.field : 0] + a.k0 + map;
          double* dst = out + (comp == 0 ? (long long)w.m * L1 + w.row0 + 2 * rbeg
                                         : (L1 - w.m) * L1 + (w.row0 - w.m) + 2 * rbeg) * a.ld;
#pragma unroll
          for (int j = 0; j < 64; ++j) {
            if (j >= nrow) break;
            const double v = i64_scaled((long long)(acc[j] - bias), e) * s_fac[warp][j];
            double* d = dst + (long long)(2 * j) * a.ld;
            *d = a.accumulate ? *d + v : v;
          }
        } else {
          double* dst = a.out[SPIN == 2 ? w.field : 0] +
                        (((long long)w.m * a.nnorth + w.row0 + rbeg) * a.kc + map) * 4 + comp;
          const long long rs = (long long)a.kc * 4;
          // phase 0 leaves A in the north slot; the same thread reads it back in phase 1
#pragma unroll
          for (int j = 0; j < 64; ++j) {
            if (j >= nrow) break;
            const double v = i64_scaled((long long)(acc[j] - bias), e);
            if (ph == 0) {
              dst[j * rs] = v;
            } else {
              const double A = dst[j * rs];
              dst[j * rs] = A + v;
              dst[j * rs + 2] = A - v;
            }
          }
        }
      }
    }
  }
  // the UMMA issuer waits for its last products before TMEM is released, the loader for its
  // last copies
  if (warp > kEpiThreads / 32) {
    tc::umma_commit_warp(&h.fin);
    for (uint32_t it = 0; it < tc::kWaitLimit; ++it)
      if (tc::mbar_try_wait(&h.fin, 0)) break;
  }
  if (tid == kEpiThreads) {
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

int tc_eag(int lmax) {
  const double b = std::sqrt((2.0 * lmax + 1.0) / (4.0 * M_PI)) * (1.0 + 0x1p-30);
  return std::ilogb(b) + 1;
}
int ceil_log2(long long x) {
  int b = 0;
  while ((1LL << b) < x) ++b;
  return b;
}
// Integer units: sums in digit units are below 2^12 times the sum of |row| / scale, and the 64-bit
// sum has 63 bits.  Analysis: sum over the north rings of |lambda| (spin 2: |lambda1| + |lambda2|)
// is below 0.85 nside for every l and m (tests/test_tc_bounds.py), against 2^EAG.  Synthesis: the
// sum over l of one parity of |lambda| 2^-EA(l) is below 0.4 (lmax/2 + 1) for the same reason.
int tc_bits_analysis(const fsht_plan* p) {
  return std::min(46, 51 - ceil_log2(p->nside) + tc_eag(p->lmax));
}
int tc_bits_synthesis(const fsht_plan* p) {
  return std::min(46, 51 - ceil_log2((2LL * (p->lmax / 2 + 1) + 4) / 5 + 1));
}

template <int DIR, int SPIN>
int launch_tc_gemm(const TcGemmArgs& a, cudaStream_t s) {
  FSHT_TRY(fsht_smem_limit((const void*)k_tc_gemm<DIR, SPIN>, kTcSmem));
  if (a.nunits > 0) k_tc_gemm<DIR, SPIN><<<a.nunits, kTcThreads, kTcSmem, s>>>(a);
  FSHT_LAUNCH_CHECK();
  return FSHT_OK;
}
}  // namespace

bool fsht_tc_supported(const fsht_plan* p) {
  return p->nside >= 32 && tc_bits_analysis(p) >= 38 && tc_bits_synthesis(p) >= 38;
}

int fsht_tc_tables_init(fsht_plan* p) {
  const size_t ntab = (size_t)tri_off(p->lmax + 1, p->lmax);
  FSHT_CUDA_TRY(cudaMalloc(&p->d_lamtab, sizeof(FshtLamRow) * ntab));
  if (p->pol) {
    FSHT_CUDA_TRY(cudaMalloc(&p->d_lamtab2, sizeof(FshtLamRow) * ntab));
    FSHT_CUDA_TRY(cudaMalloc(&p->d_poltab, sizeof(FshtPolRow) * ntab));
  }
  k_tc_table<<<p->lmax + 1, kTabThreads, 0, p->stream>>>(p->lmax, p->d_lamtab, p->d_lamtab2,
                                                         p->d_poltab);
  FSHT_LAUNCH_CHECK();
  return fsht_wave_tables_init(p, kStepBytes);
}

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
  a.row_bytes = tc_row_bytes(p);
  a.tab = alm1 ? p->d_lamtab2 : p->d_lamtab;
  a.WS = WS;
  a.EB = EB;
  a.flags = p->d_tcflag;
  const dim3 grid(wv[1] - wv[0], a.ngroups);
  if (alm1)
    k_tc_slice_alm<2><<<grid, 256, 0, s>>>(a);
  else
    k_tc_slice_alm<1><<<grid, 128, 0, s>>>(a);
  FSHT_LAUNCH_CHECK();
  return FSHT_OK;
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
  a.eag = tc_eag(p->lmax);
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
  a.unit_bits = dir == 0 ? tc_bits_analysis(p) : tc_bits_synthesis(p);
  a.eag = tc_eag(p->lmax);
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
