// The FP64 recursion step and the spin-2 functions, shared by the FMA kernels
// (legendre_fp64.cu) and the tensor-core form (legendre_fp64_tc.cu) so that both contract the
// same lambda1 / lambda2: near the poles they come from cancelling terms, and the reference's
// order of operations (get_plm_recursive.f90:31-125) is part of their last digits.
#pragma once
#include "common.cuh"

namespace {

__device__ __forceinline__ void rec_step(double& cur, double& prev, int& e, double a_cth,
                                         double b) {
  const double nx = a_cth * cur - b * prev;
  prev = cur;
  cur = nx;
  if (e < 0 && fabs(cur) > 0x1p300) {
    cur *= 0x1p-600;
    prev *= 0x1p-600;
    ++e;
  }
}

// Spin-2 lambda1/lambda2 from lambda_l (cur) and lambda_{l-1} (prev) on one ring
// (get_plm_recursive.f90:101-125).
struct PolRing {
  double cth, b_w, two_on_s2, c_w, diag1, diag2;
};
__device__ __forceinline__ PolRing pol_ring(double cth, double sth, int m) {
  PolRing r;
  const double s2 = sth * sth;
  r.cth = cth;
  r.b_w = cth / s2;
  r.two_on_s2 = 2.0 / s2;
  r.c_w = (double)m / s2;
  r.diag1 = 0.5 - 1.0 / s2;
  r.diag2 = cth / s2;
  return r;
}
__device__ __forceinline__ double normal_l(int l) {
  if (l < 2) return 0.0;
  return 1.0 / sqrt((double)(l + 2) * (double)(l + 1) * (double)l * (double)(l - 1));
}
__device__ __forceinline__ double lam_fact(int l, int m) {
  const int m1 = m > 1 ? m : 1;
  if (l <= m1) return 0.0;
  return 2.0 * sqrt((double)(2 * l + 1) / (double)(2 * l - 1) * (double)((long long)l * l - (long long)m * m));
}
// The ring-independent factors of step l (integers, exact in FP64; nm = 2 m (1 - m) at l = m).
struct PolL {
  double lm, ll, l1, nm;
  bool diag;
};
__device__ __forceinline__ PolL pol_l(int l, int m) {
  PolL p;
  p.lm = (double)((long long)l - (long long)m * m);
  p.ll = (double)l * ((double)l - 1.0);
  p.l1 = (double)l - 1.0;
  p.nm = (double)(2LL * m * (1 - m));
  p.diag = l == m;
  return p;
}
__device__ __forceinline__ void pol_lambda(const PolRing& r, const PolL& p, double cur, double prev,
                                           double lf, double nl, double& l1, double& l2) {
  if (p.diag) {
    const double nm = p.nm * nl;
    l1 = nm * cur * r.diag1;
    l2 = nm * cur * r.diag2;
  } else {
    l1 = (prev * lf * r.b_w - cur * (r.two_on_s2 * p.lm + p.ll)) * nl;
    l2 = (prev * lf - cur * (2.0 * r.cth * p.l1)) * r.c_w * nl;
  }
}
// The same without the factor N_l.
__device__ __forceinline__ void pol_lambda_raw(const PolRing& r, const PolL& p, double cur,
                                               double prev, double lf, double& l1, double& l2) {
  if (p.diag) {
    l1 = p.nm * cur * r.diag1;
    l2 = p.nm * cur * r.diag2;
  } else {
    l1 = prev * lf * r.b_w - cur * (r.two_on_s2 * p.lm + p.ll);
    l2 = (prev * lf - cur * (2.0 * r.cth * p.l1)) * r.c_w;
  }
}

}  // namespace
