// Exact rounding of the tensor-core update's level sums to FP64, written once for the device and the host
// (the host build is what the CPU tests check against the FP64 expression it replaces).
#pragma once
#include <stdint.h>
#include <string.h>
#include <math.h>

#ifdef __CUDACC__
#define SKN_HD __host__ __device__ __forceinline__
#else
#define SKN_HD inline
#endif

SKN_HD int skn_clz64(unsigned long long x) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)x);
#else
  return __builtin_clzll(x);
#endif
}

SKN_HD double skn_bits_to_double(unsigned long long b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double d;
  memcpy(&d, &b, sizeof d);
  return d;
#endif
}

// The double nearest to (hi * 2^21 + lo) * 2^e, ties to even, assembled with integer operations: the exact
// sum is formed in 128 bits, its top 53 bits are rounded and packed with the exponent.  It equals
// fma((double)hi, 2^-35, (double)lo * 2^-56) * 2^(e + 56), one rounding of the same exact value, for
// |hi| < 2^53 and |lo| < 2^53, while keeping the int64-to-FP64 conversions and the scaling off the FP64 pipe.
// Results outside the normal range take that FP64 expression.
SKN_HD double exact_to_double(long long hi, long long lo, int e) {
  const __int128 v = ((__int128)hi << 21) + (__int128)lo;
  if (v == 0) return 0.0;
  const unsigned long long sgn = v < 0 ? 0x8000000000000000ull : 0ull;
  const unsigned __int128 a = v < 0 ? (unsigned __int128)(-v) : (unsigned __int128)v;
  const unsigned long long ah = (unsigned long long)(a >> 64), al = (unsigned long long)a;
  int msb = ah ? 127 - skn_clz64(ah) : 63 - skn_clz64(al);   // a in [2^msb, 2^(msb+1))
  unsigned long long m;                                       // 53-bit significand
  if (msb > 52) {
    const int sh = msb - 52;
    m = (unsigned long long)(a >> sh);
    const unsigned __int128 rem = a - ((unsigned __int128)m << sh);
    const unsigned __int128 half = (unsigned __int128)1 << (sh - 1);
    if (rem > half || (rem == half && (m & 1ull))) {
      ++m;
      if (m == (1ull << 53)) {
        m >>= 1;
        ++msb;
      }
    }
  } else {
    m = (unsigned long long)(a << (52 - msb));
  }
  const int be = msb + e + 1023;                              // value = m * 2^(msb - 52 + e), m in [2^52, 2^53)
  if (be <= 0 || be >= 2047) return fma((double)hi, 0x1p-35, (double)lo * 0x1p-56) * ldexp(1.0, e + 56);
  return skn_bits_to_double(sgn | ((unsigned long long)be << 52) | (m & 0xFFFFFFFFFFFFFull));
}

// The double nearest to (hi * 2^28 + lo) * 2^e (ties away from zero), for |hi| < 2^46 and |lo| < 2^46: the sum is
// normalised in 64 bits (its 53 leading bits and one rounding increment), about 30 integer instructions.
SKN_HD double round_sum28(long long hi, long long lo, int e) {
  long long h = hi + (lo >> 28);
  unsigned long long l = (unsigned long long)lo & 0xFFFFFFFull;
  const bool neg = h < 0;
  if (neg) {                                                  // negate the pair: l stays in [0, 2^28)
    h = -h - (l != 0);
    l = (0x10000000ull - l) & 0xFFFFFFFull;
  }
  const int lz = h ? skn_clz64((unsigned long long)h) - 11 : 53;
  const int k = lz < 28 ? lz : 28;                            // bits of l that still fit below 53
  const int d = 28 - k;
  unsigned long long t = ((unsigned long long)h << k) + ((l + ((1ull << d) >> 1)) >> d);
  if (t == 0) return 0.0;
  int s = skn_clz64(t) - 11;                                  // below 2^52 only when k = 28: exact shift
  s = s < 0 ? 0 : s;                                          // t = 2^53 after rounding up: carries into the exponent
  t <<= s;
  const int be = 1075 + d - s + e;                            // value = t 2^(d - s + e), t in [2^52, 2^53]
  if (be <= 0 || be >= 2046) return ldexp((double)(neg ? -(long long)t : (long long)t), d - s + e);
  return skn_bits_to_double((neg ? 0x8000000000000000ull : 0ull) + ((unsigned long long)be << 52) +
                            (t - 0x10000000000000ull));
}

// The double nearest to (h * 2^28 + m) * 2^k for any |h| < 2^62 and |m| < 2^62 (ties away from zero, but for bits of m
// below 2^-64 of the sum): the sum is normalised in 64 bits. About 30 integer instructions and no FP64 one.
SKN_HD double round_wide28(long long h, long long m, int k) {
  long long H = h + (m >> 28);
  unsigned long long l = (unsigned long long)m & 0xFFFFFFFull;
  const bool neg = H < 0;
  if (neg) {                                                  // negate the pair: l stays in [0, 2^28)
    H = -H - (l != 0);
    l = (0x10000000ull - l) & 0xFFFFFFFull;
  }
  k += 28;
  if (H == 0) {
    H = (long long)l;
    l = 0;
    k -= 28;
    if (H == 0) return 0.0;
  }
  const int z = skn_clz64((unsigned long long)H);             // 1 .. 63
  const unsigned long long top = ((unsigned long long)H << z) | ((l << 36) >> (64 - z));
  const unsigned long long t = (top >> 11) + ((top >> 10) & 1);   // in [2^52, 2^53]: rounding up carries into the exponent
  const int be = 1086 - z + k;                                // value = t 2^(11 - z + k)
  if (be <= 0 || be >= 2046) return ldexp((double)(neg ? -(long long)t : (long long)t), 11 - z + k);
  return skn_bits_to_double((neg ? 0x8000000000000000ull : 0ull) + ((unsigned long long)be << 52) + (t - 0x10000000000000ull));
}

// a / b from b's rounded reciprocal: the product corrected by its remainder (Markstein, IBM J. Res. Dev. 34, 1990), which
// leaves the quotient's own rounding for normal operands.  An infinite or NaN product is the quotient.
SKN_HD double skn_quotient(double a, double b, double inv_b) {
  const double q = a * inv_b;
  const double c = fma(fma(-q, b, a), inv_b, q);
#ifdef __CUDA_ARCH__
  return (__double2hiint(q) & 0x7fffffff) < 0x7ff00000 ? c : q;      // not on the FP64 pipe
#else
  return fabs(q) <= 1.7976931348623157e308 ? c : q;
#endif
}

// 1 / b to twice the working precision (the remainder of the reciprocal is exact), and a / b by it for finite a: the two
// products are rounded together, so the result is off by its own rounding alone.  Two instructions where many a share a b.
struct SknRecip {
  double hi, lo;
};
SKN_HD SknRecip skn_recip(double b) {
  const double hi = 1.0 / b;
  return {hi, fma(-hi, b, 1.0) * hi};
}
SKN_HD double skn_over(double a, SknRecip r) { return fma(a, r.hi, a * r.lo); }
