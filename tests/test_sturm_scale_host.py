"""The exponent shift of the tridiagonal eigenvalue search (csrc/sturm.cuh), built for the host: bit for bit ldexp where the
result is normal, an infinity above, truncated below the normal range, subnormal inputs included; and the search at the
ends of the range that its squared couplings allow."""
import os
import shutil
import subprocess

import numpy as np
import pytest
import scipy.linalg as sla

from conftest import ROOT
from test_sturm_host import SHIM, search  # noqa: F401  (the fixture)

CHECK = r"""
#include <cstdio>
#include <cstdint>
#include "sturm.cuh"
int main() {
  uint64_t x = 88172645463325252ull;
  auto next = [&]() { x ^= x << 13; x ^= x >> 7; x ^= x << 17; return x; };
  long bad = 0, n = 0;
  auto test = [&](double v, int s) {
    const double got = skn_sturm::shift_exp(v, s), want = std::ldexp(v, s);
    ++n;
    if (v != v) { bad += got == got; return; }
    if (std::fpclassify(want) == FP_SUBNORMAL || (want == 0.0 && v != 0.0) || std::fabs(want) == 0x1p-1022) {
      // cut off below the last place, of the right sign
      bad += !(std::fabs(got - want) <= 4.95e-324 && std::signbit(got) == std::signbit(v));
      return;
    }
    bad += std::memcmp(&got, &want, 8) != 0;
  };
  for (int i = 0; i < 2000000; ++i) {
    uint64_t b = next();
    if (i % 3 == 0) b &= 0x800fffffffffffffull;                    // subnormal
    if (i % 7 == 0) b &= 0x8000000000000000ull | (next() & 0xff);  // the smallest of them, and zeros
    double v;
    std::memcpy(&v, &b, 8);
    test(v, (int)(next() % 2200) - 1100);
  }
  const double edge[] = {0.0, -0.0, 4.95e-324, -4.95e-324, 0x1p-1022, 0x1.fffffffffffffp1023, -0x1p1023, INFINITY, -INFINITY, NAN};
  for (double v : edge)
    for (int s = -1100; s <= 1100; ++s) test(v, s);
  std::printf("%ld of %ld\n", bad, n);
  return bad != 0;
}
"""


def test_shift_is_ldexp_at_every_edge(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    shutil.copy(os.path.join(ROOT, "slakonet_gb300", "csrc", "sturm.cuh"), tmp_path)
    (tmp_path / "skn_common.cuh").write_text(SHIM)
    (tmp_path / "check.cpp").write_text(CHECK)
    exe = str(tmp_path / "check")
    subprocess.check_call([cxx, "-O2", "-std=c++17", "-w", str(tmp_path / "check.cpp"), "-o", exe])
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


@pytest.mark.parametrize("k", [-505, -480, 400, 505])      # the couplings' squares stay in the normal range
def test_search_at_extreme_scales(search, k):              # noqa: F811
    rng = np.random.default_rng(k + 600)
    for n in (2, 17, 90):
        d, e = rng.standard_normal(n), rng.standard_normal(n - 1)
        ref = sla.eigvalsh_tridiagonal(d, np.abs(e))
        got = search(d * 2.0 ** k, (e * 2.0 ** k) ** 2) * 2.0 ** -k
        norm = np.abs(ref).max()
        assert np.abs(got - ref).max() <= (1e-14 + 10 * 2.2e-16) * 3.0 * norm
