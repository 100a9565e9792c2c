// Integer units of the FP64 digit products (legendre_fp64_tc.cu), in plain C++ so that host tests
// can check them against the sums.
//
// Operands are 62-bit fixed-point numbers against a power-of-two scale; in the weight of the two
// leading digits' product a product of two operands is below 2^12.  A sum of products of at most S
// times that leaves the kernel as a 64-bit integer of unit 2^-bits, so S 2^(12 + bits) <= 2^63 has to
// hold (tests/test_tc_units.py).
#pragma once
#include <algorithm>
#include <cmath>

struct FshtTcUnits {
  int bits;      // unit 2^-bits; the drains take 40..46
  int head;      // spare bits of the columns in place of units below 40: |v| < 2^(E - head) for the
                 // column exponent E
};
inline FshtTcUnits fsht_tc_units_of(int bits) {
  return FshtTcUnits{std::min(46, std::max(40, bits)), std::max(0, 40 - bits)};
}

inline int fsht_ceil_log2(long long x) {
  int b = 0;
  while ((1LL << b) < x) ++b;
  return b;
}

// Exponent of the lambda rows of the analysis: 2^eag > sqrt((2 lmax + 1) / 4 pi).
inline int fsht_tc_eag(int lmax) {
  const double b = std::sqrt((2.0 * lmax + 1.0) / (4.0 * 3.14159265358979323846)) * (1.0 + 0x1p-30);
  return std::ilogb(b) + 1;
}
// Analysis: sum over the north rings of |lambda| (spin 2: |lambda1| + |lambda2|) is below 0.85 nside
// for every l and m (tests/test_tc_bounds.py), against 2^eag.
inline FshtTcUnits fsht_tc_units_analysis(int nside, int lmax) {
  return fsht_tc_units_of(51 - fsht_ceil_log2(nside) + fsht_tc_eag(lmax));
}
// Synthesis: the parities are added and subtracted, lmax + 1 - m products with rows and columns
// below one.  (Over l, |lambda| 2^-EA(l) has no smaller average that holds for every lmax: at the
// polar ring lambda_l0 stays near its maximum up to l of about nside, and columns of one sign reach
// 0.82 of the bound.)
inline FshtTcUnits fsht_tc_units_synthesis(int lmax) {
  return fsht_tc_units_of(51 - fsht_ceil_log2(lmax + 1));
}
// Sizes of the digit contraction.  (lmax above 5113, at nside 2048, has not been measured.)
inline bool fsht_tc_sizes(int nside, int lmax) {
  return nside >= 32 && lmax <= 5113 && fsht_tc_units_analysis(nside, lmax).head == 0;
}
// Ring transforms: sums of at most nk <= q + 1 products against the cosines' 2^1; 2^extra of them
// (north and south, or the four mirrored samples) are added and subtracted.
inline FshtTcUnits fsht_tc_units_dft(int nk, int extra) {
  return fsht_tc_units_of(51 - extra - fsht_ceil_log2((nk + 1) / 2));
}
