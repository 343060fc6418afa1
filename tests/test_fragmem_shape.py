"""The fragment-memory kernel's default launch shape (awsem_shape.h): every
separation in one unit, enough units to fill the multiprocessors, and no more
than they need however many separations a table reaches over."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = r"""
#include <cstdio>
#include "awsem_shape.h"
using namespace awsem;
int main()
{
  const int sms = 148;
  for (int nd = 0; nd <= 64; nd++)
    for (int g = 0; g < 70000; g += g < 300 ? 1 : 37) {
      const FMShape d = fm_shape(true, g, nd, sms), m = fm_shape(false, g, nd, sms);
      const long long n = nd > 1 ? nd : 1, groups = g > 1 ? g : 1;
      bool ok = d.dsplit >= 1 && d.dsplit <= n && m.dsplit >= 1 && m.dsplit <= n && d.grid == 0;
      ok = ok && (d.dsplit == n || groups * d.dsplit >= 96 * sms) && (m.dsplit == n || groups * m.dsplit >= 16 * sms);
      ok = ok && groups * (d.dsplit - 1) < 96 * sms && groups * (m.dsplit - 2) < 16 * sms;
      ok = ok && m.dsplit >= (n > 1 ? 2 : 1) && m.grid == (32 * groups <= 65536 ? 2 : 3) * sms;
      if (!ok) return printf("%d groups of %d: %d, %d by %d\n", g, nd, d.dsplit, m.dsplit, m.grid), 1;
    }
  return 0;
}
"""


def test_shapes(tmp_path):
    (tmp_path / "t.cpp").write_text(CODE)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "awsemmd_b200", "csrc"), "-o", exe, str(tmp_path / "t.cpp")],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
