// Host build of the tridiagonal eigenvalue search (slakonet_gb300/csrc/sturm.cuh, copied beside this file together with a
// skn_common.cuh of what it needs): reads n, the diagonal and the squared off-diagonal, prints the n eigenvalues.
#include <cstdio>
#include <vector>

#include "sturm.cuh"

int main() {
  int n;
  while (std::scanf("%d", &n) == 1) {
    std::vector<double> d(n), e2(n);
    std::vector<float> d32(n), e232(n);
    for (int i = 0; i < n; ++i)
      if (std::scanf("%lf", &d[i]) != 1) return 1;
    for (int i = 0; i + 1 < n; ++i)
      if (std::scanf("%lf", &e2[i]) != 1) return 1;
    double lo = 1e300, hi = -1e300, emax = 0.0;
    for (int i = 0; i < n; ++i) {
      const double ea = i > 0 ? sqrt(e2[i - 1]) : 0.0, eb = i + 1 < n ? sqrt(e2[i]) : 0.0;
      lo = fmin(lo, d[i] - ea - eb);
      hi = fmax(hi, d[i] + ea + eb);
      emax = fmax(emax, e2[i]);
      d32[i] = (float)d[i];
      e232[i] = (float)e2[i];
    }
    const skn_sturm::Bounds B = skn_sturm::make_bounds(lo, hi, emax, n);
    for (int j = 0; j < n; ++j) std::printf("%.17g ", skn_sturm::eigenvalue(d.data(), e2.data(), d32.data(), e232.data(), n, j, B));
    std::printf("\n");
  }
}
