// Eigenvalues of a real symmetric tridiagonal matrix (diagonal d, squared
// off-diagonal e2, e2[i] coupling rows i and i+1), one eigenvalue per thread.
// Shared by the one-CTA and the cluster eigensolvers.
//
//  1. FP32 trisection on the rounded matrix brackets eigenvalue j to ~1e-6 of
//     the spectrum's scale (FP32 runs 64x faster than FP64 on GB300).
//  2. The bracket is widened by a margin covering the FP32 rounding and
//     checked with two FP64 Sturm counts (else the Gershgorin interval is used).
//  3. If it holds eigenvalue j alone, safeguarded secant steps on the
//     characteristic polynomial p(x) = det(T - x I) finish it: the two counts of
//     step 2 already give p at the bracket's ends, each step also yields the Sturm
//     count at the new point, which keeps the bracket, and a step that leaves the
//     bracket is replaced by bisection.  Over a bracket of 4e-6 of the scale p is
//     nearly linear, so two more evaluations (three FP64 operations per row, against
//     five for one with the derivative) replace ~28 bisection steps.
//  4. Clustered or degenerate eigenvalues (the bracket holds several) are
//     bisected in FP64 to 2e-15 of the scale.
#pragma once
#include "skn_common.cuh"

namespace skn_sturm {
namespace {   // internal linkage: every including file gets its own copy

__device__ __forceinline__ int sign_bit(double v) { return (int)((unsigned long long)__double_as_longlong(v) >> 63); }

// Exponent field of |v| (biased), for power-of-two rescaling.
__device__ __forceinline__ int exp_field(double v) { return (int)((__double_as_longlong(v) >> 52) & 0x7ff); }

__device__ __forceinline__ int clz64(unsigned long long v) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)v);
#else
  return __builtin_clzll(v);
#endif
}
// v 2^s where v, or the result, is subnormal or out of range: what falls below is cut off, what exceeds is infinite.
__device__ inline double shift_exp_edge(double v, int s) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v), sign = b & 0x8000000000000000ull;
  const int e = (int)((b >> 52) & 0x7ff);
  unsigned long long f = b & 0xfffffffffffffull;
  if (e == 0x7ff || (e == 0 && f == 0)) return v;
  const int z = e == 0 ? clz64(f) - 11 : 0;
  f = e == 0 ? f << z : f | 0x10000000000000ull;
  const int t = (e == 0 ? 1 - z : e) + s;
  if (t >= 0x7ff) return __longlong_as_double((long long)(sign | 0x7ff0000000000000ull));
  if (t <= 0) return __longlong_as_double((long long)(sign | (t > -52 ? f >> (1 - t) : 0)));
  return __longlong_as_double((long long)(sign | ((unsigned long long)t << 52) | (f & 0xfffffffffffffull)));
}
// v 2^s by its exponent field, so that the rescaling below, which a compiler may execute on every step, stays off the
// FP64 pipe.
__device__ __forceinline__ double shift_exp(double v, int s) {
  const int h = __double2hiint(v), e = (h >> 20) & 0x7ff, t = e + s;
  if (e != 0 && e != 0x7ff && t > 0 && t < 0x7ff) return __hiloint2double(h + (int)((unsigned)s << 20), __double2loint(v));
  return shift_exp_edge(v, s);
}

// Number of eigenvalues below x: sign changes of the determinant sequence
// p_i = (d_i - x) p_{i-1} - e2_{i-1} p_{i-2} (three FP64 operations per step, no
// division).  (p, p_prev) are rescaled by exact powers of two when p's exponent
// drifts, and an exact zero p_i takes the sign opposite to p_{i-1} (the tiny
// negative pivot LAPACK substitutes).
__device__ __forceinline__ int count64(const double* d, const double* e2, int n, double x) {
  double pm = 1.0, p = d[0] - x;
  if (is_zero_bits(p)) p = -0x1p-200;
  int c = sign_bit(p);
  int sp = c;
  for (int i = 1; i < n; ++i) {
    double pn = fma(-e2[i - 1], pm, (d[i] - x) * p);
    if (is_zero_bits(pn)) pn = flip_sign(p) * 0x1p-200;
    const int sn = sign_bit(pn);
    c += sn ^ sp;
    sp = sn;
    pm = p;
    p = pn;
    const int ex = exp_field(p);
    if (ex > 1023 + 480 || ex < 1023 - 480) {
      p = shift_exp(p, 1023 - ex);
      pm = shift_exp(pm, 1023 - ex);
    }
  }
  return c;
}

// The same count plus the polynomial's value p(x) = p 2^e.
__device__ __forceinline__ int count_value64(const double* d, const double* e2, int n, double x, double& val, int& e) {
  double pm = 1.0, p = d[0] - x;
  e = 0;
  if (is_zero_bits(p)) p = -0x1p-200;
  int c = sign_bit(p);
  int sp = c;
  for (int i = 1; i < n; ++i) {
    double pn = fma(-e2[i - 1], pm, (d[i] - x) * p);
    if (is_zero_bits(pn)) pn = flip_sign(p) * 0x1p-200;
    const int sn = sign_bit(pn);
    c += sn ^ sp;
    sp = sn;
    pm = p;
    p = pn;
    const int ex = exp_field(p);
    if (ex > 1023 + 480 || ex < 1023 - 480) {
      p = shift_exp(p, 1023 - ex);
      pm = shift_exp(pm, 1023 - ex);
      e += ex - 1023;
    }
  }
  val = p;
  return c;
}

// Zero of the line through (x0, p0 2^e0) and (x1, p1 2^e1), as a step from x1.
__device__ __forceinline__ double secant_step(double x0, double p0, int e0, double x1, double p1, int e1) {
  const int de = min(max(e0 - e1, -1000), 1000);
  const double s = p0 * (1.0 / p1) * __longlong_as_double((long long)(1023 + de) << 52);
  return (x1 - x0) * (1.0 / (s - 1.0));
}

// FP32 counts at x0 < x1 on the rounded tridiagonal (LDL^T pivots).  The bracket they give is checked in FP64, so the
// quotient's last bits do not matter: an approximate reciprocal.  A step is one chain of about 50 clocks; two chains side
// by side cost little more than one while a partition has few warps.
__device__ __forceinline__ float recip32(float q) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(q));
  return r;
#else
  return 1.0f / q;
#endif
}
__device__ __forceinline__ void count32(const float* d, const float* e2, int n, float x0, float x1, float pivmin, int& c0,
                                        int& c1) {
  float q0 = d[0] - x0, q1 = d[0] - x1;
  if (fabsf(q0) < pivmin) q0 = -pivmin;              // before it is counted: a zero counted as positive and carried on as
  if (fabsf(q1) < pivmin) q1 = -pivmin;              // negative loses an eigenvalue
  c0 = q0 < 0.0f;
  c1 = q1 < 0.0f;
#pragma unroll 4
  for (int i = 1; i < n; ++i) {
    const float di = d[i], ei = e2[i - 1];
    q0 = fmaf(-ei, recip32(q0), di - x0);
    q1 = fmaf(-ei, recip32(q1), di - x1);
    if (fabsf(q0) < pivmin) q0 = -pivmin;
    if (fabsf(q1) < pivmin) q1 = -pivmin;
    c0 += q0 < 0.0f;
    c1 += q1 < 0.0f;
  }
}

// Bounds shared by the threads of one matrix: Gershgorin interval [lo, hi]
// (already widened), FP64 target width atol, FP32 pivot floor, FP32 margin.
struct Bounds {
  double lo, hi, atol, margin;
  float pivmin32;
};

// A row's part of `emax` below: its squared coupling, infinite where that or the diagonal is an infinity or a NaN (minima
// and maxima pass over NaNs).
__device__ __forceinline__ double row_max(double d, double e2) {
  const double inf = __longlong_as_double(0x7ff0000000000000LL);
  return exp_field(d) == 0x7ff || exp_field(e2) == 0x7ff ? inf : e2;
}

// lo, hi: Gershgorin's; emax: the largest of row_max.  An infinite emax makes every eigenvalue NaN.
__device__ __forceinline__ Bounds make_bounds(double lo, double hi, double emax, int n) {
  Bounds B;
  if (exp_field(emax) == 0x7ff) lo = __longlong_as_double(0x7ff8000000000000LL);
  const double bnorm = fmax(fmax(fabs(lo), fabs(hi)), 1e-300);
  B.lo = lo - (2.2e-16 * bnorm * 4.0 * n + 1e-300);
  B.hi = hi + (2.2e-16 * bnorm * 4.0 * n + 1e-300);
  B.atol = 2e-15 * bnorm;
  B.pivmin32 = 1.1754944e-38f * fmaxf(1.0f, (float)emax);
  B.margin = 32.0 * 5.9604645e-8 * bnorm;   // covers FP32 rounding of T and of the count
  return B;
}

// Eigenvalue j (0-based, ascending) of the tridiagonal.
__device__ double eigenvalue(const double* d, const double* e2, const float* d32, const float* e232, int n, int j,
                             const Bounds& B) {
  if (!(B.lo <= B.hi)) return __longlong_as_double(0x7ff8000000000000LL);
  float a32 = (float)B.lo, b32 = (float)B.hi;
  const float enough = 0.25f * (float)B.margin;      // the bracket is widened by the margin anyway
  for (int it = 0; it < 26 && b32 - a32 > enough; ++it) {
    const float third = (b32 - a32) * (1.0f / 3.0f), x0 = a32 + third, x1 = b32 - third;
    if (!(x0 > a32 && x1 < b32 && x0 < x1)) break;
    int c0, c1;
    count32(d32, e232, n, x0, x1, B.pivmin32, c0, c1);
    if (c0 > j) b32 = x0;
    else if (c1 > j) { a32 = x0; b32 = x1; }
    else a32 = x1;
  }
  double a = (double)a32 - B.margin, b = (double)b32 + B.margin;
  if (a < B.lo) a = B.lo;
  if (b > B.hi) b = B.hi;
  double p0, p1;
  int e0, e1;
  const int ca = count_value64(d, e2, n, a, p0, e0);
  const int cb = count_value64(d, e2, n, b, p1, e1);
  if (!(ca <= j && cb > j)) {
    a = B.lo;
    b = B.hi;
  } else if (ca == j && cb == j + 1) {
    // eigenvalue j alone in (a, b]: safeguarded secant from the bracket's ends.  A step that leaves the
    // bracket, or is not at least halving the previous step, is replaced by bisection, so the bracket keeps
    // shrinking.
    // A line through the ends can point at an eigenvalue outside, when an end all but touches it: p is then as good as
    // zero there, its step vanishes and would pass for convergence.  The bracket leaves its own eigenvalue well inside, so
    // that shows as ends of very different size, and such an eigenvalue is taken only where the counts change.
    const bool plain = abs((exp_field(p0) + e0) - (exp_field(p1) + e1)) <= 6;
    double x1 = b, xn = b + secant_step(a, p0, e0, b, p1, e1);
    double dx_old = b - a;
    for (int it = 0; it < 16; ++it) {
      if (!(xn > a && xn < b)) xn = 0.5 * (a + b);
      const double x = xn;
      double p2;
      int e2x;
      const int c = count_value64(d, e2, n, x, p2, e2x);
      if (c > j) b = x; else a = x;
      if (b - a <= B.atol) break;
      const double step = secant_step(x1, p1, e1, x, p2, e2x);
      x1 = x;
      p1 = p2;
      e1 = e2x;
      xn = x + step;
      // converged: the last step may land on the bracket's edge (the root lies within rounding of
      // the point just counted), so it is tested before the bracket, not after
      if (fabs(step) <= B.atol && xn >= a && xn <= b) {
        if (plain || (count64(d, e2, n, xn - 2.0 * B.atol) <= j && count64(d, e2, n, xn + 2.0 * B.atol) > j)) return xn;
        xn = a - 1.0;                                // bisect
      }
      if (xn > a && xn < b && fabs(step) <= 0.5 * dx_old) {
        dx_old = fabs(step);
      } else {
        dx_old = 0.5 * (b - a);
        xn = 0.5 * (a + b);
      }
    }
  }
  for (int it = 0; it < 200 && (b - a) > B.atol; ++it) {
    const double mid = 0.5 * (a + b);
    if (mid <= a || mid >= b) break;
    if (count64(d, e2, n, mid) > j) b = mid; else a = mid;
  }
  return 0.5 * (a + b);
}

}  // namespace
}  // namespace skn_sturm
