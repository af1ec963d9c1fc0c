// Host check of skn_quotient and skn_over (slakonet_gb300/csrc/exact_round.cuh).  The first is bit for bit a / b, on random
// operands of the Fermi search's range, on near-halfway quotients, and on zeros, infinities and NaNs; the second within
// 0.501 units of the last place of it for finite operands.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>

#include "exact_round.cuh"

int main(int argc, char** argv) {
  const long long cases = argc > 1 ? atoll(argv[1]) : 2000000;
  std::mt19937_64 g(20261205);
  std::uniform_real_distribution<double> u(1.0, 2.0);
  long long bad = 0;
  auto test = [&](double a, double b) {
    const double got = skn_quotient(a, b, 1.0 / b), want = a / b;
    if (want != want ? got == got : std::memcmp(&got, &want, 8) != 0) {
      if (want == 0.0 && got == 0.0) return;                     // a zero of either sign
      if (bad++ < 5) std::printf("%a / %a: %a, not %a\n", a, b, got, want);
    }
  };
  auto over = [&](double a, double b) {
    const double got = skn_over(a, skn_recip(b));
    const long double want = (long double)a / b;
    const double ulp = std::nextafter(std::fabs((double)want), INFINITY) - std::fabs((double)want);
    if (!(std::fabs((double)(got - want)) <= 0.501 * ulp) && bad++ < 5) std::printf("over %a / %a: %a\n", a, b, got);
  };
  const double kT[] = {0.01, 0.0137, 0.025 / 27.211, 1e-3, 0.3, 1.0, 3.0, 1e-8, 1e6};
  for (long long i = 0; i < cases; ++i) {
    const double b = i % 3 ? kT[g() % 9] : std::ldexp(u(g), (int)(g() % 200) - 100);
    double a = std::ldexp(g() & 1 ? u(g) : -u(g), (int)(g() % 200) - 100);
    if (i % 5 == 0) a = std::nextafter(b * u(g), g() & 1 ? 1e300 : -1e300);
    test(a, b);
    over(a, b);
  }
  const double edge[] = {0.0, -0.0, INFINITY, -INFINITY, NAN, 1e300, -1e300};
  for (double b : kT)
    for (double a : edge) test(a, b);
  std::printf("%lld mismatches in %lld\n", bad, cases);
  return bad != 0;
}
