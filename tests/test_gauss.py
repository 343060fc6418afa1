"""FP64 Gaussians of the fragment-memory term (awsem_gauss.h, the kernel's own
operations compiled for the host) against 80-bit arithmetic."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# The function: one rounding (half a unit in the last place, at most 2^-53 of
# the value), and in units of 2^-53: 0.011 for that of the polynomial's last
# step (its result is at most 0.0109), as much for the step before, 0.04 for the
# Taylor remainder, 2^-20 for the low parts.  The row factor: half a unit, and
# 2^-20 of one for its correction.
CODE = r"""
#include <cmath>
#include <cstdio>
#include <limits>
#include "awsem_gauss.h"
using namespace awsem::dev;
int main()
{
  const long double ln2 = 0.693147180559945309417232121458176568L;
  unsigned long long r = 88172645463325252ull;
  auto rnd = [&] { r ^= r << 13; r ^= r >> 7; r ^= r << 17; return (double) (r >> 11) * 0x1p-53; };
  for (int k = 0; k < 400000; k++) {
    const double z = -(k % 4 == 0 ? rnd() : k % 4 == 1 ? 40 * rnd() : 1000 * rnd());
    const long double x = (long double) z * ln2 / 32, want = expl(x);
    const long double err = fabsl(gauss_host(z) - want) / want * 0x1p53L;
    if (err > 1.08L + fabsl(x) * 0x1p-9L) return printf("z %a: %Lg units\n", z, err), 1;
  }
  for (int k = 0; k < 200000; k++) {
    const double s2 = k < 64 ? pow((double) k + 1, 0.3) : exp(40 * rnd() - 20);
    const long double want = -32 / (ln2 * 2 * (long double) s2), got = gauss_factor(s2);
    int e;
    frexp((double) got, &e);
    const long double err = fabsl(got - want) / ldexpl(1.0L, e - 53);
    if (err > 0.5L + 0x1p-9L) return printf("s2 %a: %Lg units in the last place\n", s2, err), 1;
  }
  const double inf = std::numeric_limits<double>::infinity();
  if (gauss_host(0.0) != 1.0 || gauss_host(-1e59) != 0.0 || gauss_host(-inf) != 0.0) return printf("ends\n"), 1;
  if (gauss_factor(0.0) != -inf || gauss_factor(1e-310) != -inf || gauss_factor(inf) != 0.0) return printf("factor's ends\n"), 1;
  return 0;
}
"""


def test_gaussian_and_factor(tmp_path):
    (tmp_path / "t.cpp").write_text(CODE)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-I", os.path.join(ROOT, "awsemmd_b200", "csrc"), "-o", exe,
                    str(tmp_path / "t.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
