// Host check of round_sum28 (slakonet_gb300/csrc/exact_round.cuh) against 128-bit integer arithmetic: the nearest
// double of (hi 2^28 + lo) 2^e, ties away from zero, on random pairs, cancelling pairs and near-ties.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>

#include "exact_round.cuh"

static double nearest(__int128 v, int e) {
  const bool neg = v < 0;
  unsigned __int128 m = neg ? -(unsigned __int128)v : (unsigned __int128)v;
  int up = 0;
  while ((m >> up) >= ((unsigned __int128)1 << 54)) ++up;       // 54 bits: 53 and the rounding bit
  if ((m >> up) >= ((unsigned __int128)1 << 53)) ++up;
  if (up) m = (m + ((unsigned __int128)1 << (up - 1))) >> up;
  const double r = std::ldexp((double)(unsigned long long)m, up + e);
  return neg ? -r : r;
}

int main(int argc, char** argv) {
  const long long cases = argc > 1 ? atoll(argv[1]) : 2000000;
  std::mt19937_64 g(20261205);
  long long bad = 0;
  for (long long it = 0; it < cases; ++it) {
    long long hi = (long long)(g() >> 17) - (1ll << 46);        // |hi| <= 2^46
    long long lo = (long long)(g() >> 17) - (1ll << 46);
    switch (it % 6) {
      case 1: hi >>= (g() % 46); break;
      case 2: hi = 0; lo >>= (g() % 46); break;
      case 3: hi = (long long)(g() % 5) - 2; break;
      case 4: lo = -(hi << 17 >> 17) ; break;
      case 5: lo = (1ll << 27) * ((long long)(g() % 3) - 1) + (long long)(g() % 3) - 1; break;   // near-ties
      default: break;
    }
    const int e = (int)(g() % 200) - 100;
    const double ref = nearest(((__int128)hi << 28) + lo, e), got = round_sum28(hi, lo, e);
    if (ref != got) {
      if (bad < 5) std::printf("hi=%lld lo=%lld e=%d: expected %.17g, got %.17g\n", hi, lo, e, ref, got);
      ++bad;
    }
  }
  for (long long it = 0; it < cases; ++it) {                    // round_wide28: within a unit of 2^-64 of the tie
    long long h = (long long)(g() >> 1) - (1ll << 62), m = (long long)(g() >> 1) - (1ll << 62);
    if (it % 3) h >>= (g() % 63);
    if (it % 2) m >>= (g() % 63);
    if (it % 7 == 0) h = (long long)(g() % 3) - 1;
    if (it % 7 == 1) m = -(h << 28);
    const int e = (int)(g() % 200) - 100;
    const __int128 v = ((__int128)h << 28) + m;
    const double got = round_wide28(h, m, e), ref = nearest(v, e);
    const double off = std::fabs((double)(v - (__int128)std::ldexp(got, -e)));
    const double ulp = std::ldexp(1.0, std::ilogb(v ? (double)v : 1.0) - 52);
    if (ref != got && !(v != 0 && off <= 0.5001 * ulp)) {
      if (bad < 5) std::printf("wide h=%lld m=%lld e=%d: expected %.17g, got %.17g\n", h, m, e, ref, got);
      ++bad;
    }
  }
  std::printf("%lld mismatches in %lld cases\n", bad, cases);
  return bad != 0;
}
