"""The cell grid's shape and coordinates (awsem_grid.h, the kernel's own code
compiled for the host): every box, ordinary or made huge or empty by positions
out of range, gets at most the cells there is room for, and every coordinate a
cell of them."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = r"""
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <limits>
#include "awsem_grid.h"
using namespace awsem::dev;
int main()
{
  const float inf = std::numeric_limits<float>::infinity(), nan = std::numeric_limits<float>::quiet_NaN();
  const float at[] = {-inf, -3e38f, -1e30f, -1e12f, -2.3e9f, -1e5f, -300.f, 0.f, 17.f, 300.f, 1e5f, 2.3e9f, 1e12f, 1e30f, 3e38f, inf, nan};
  const float radius[] = {1e-3f, 12.f, 18.f, 1e6f, 1e30f, 3e38f, inf};
  const int caps[] = {64, 4098, 80000, 2000000};
  long long boxes = 0;
  for (float l0 : at) for (float h0 : at) for (float l1 : at) for (float h1 : {-inf, 0.f, 40.f, 2.1e9f, inf}) for (float r : radius) for (int cap : caps) {
    const float lo[3] = {l0, l1, -30.f}, hi[3] = {h0, h1, 1e10f};
    float cell = r;
    int n[3];
    grid_shape(lo, hi, cap, cell, n);
    const long long tot = (long long) n[0] * n[1] * n[2];
    if (n[0] < 1 || n[1] < 1 || n[2] < 1 || tot > cap) return printf("shape %g %g %g %g cell %g: %d %d %d\n", l0, h0, l1, h1, cell, n[0], n[1], n[2]), 1;
    for (int k = 0; k < 2; k++)
      for (float p : at) {
        const int c = grid_coord(p, lo[k], 1.f / cell, n[k]);
        if (c < 0 || c >= n[k]) return printf("coordinate %g from %g cell %g of %d: %d\n", p, lo[k], cell, n[k], c), 1;
      }
    boxes++;
  }
  // ordinary boxes: the widths counted in 32 bits, as before
  for (int k = 0; k < 2000; k++) {
    const float lo[3] = {-200.f + k, -100.f, 3.f * k}, hi[3] = {lo[0] + 0.37f * k, 250.f, lo[2] + 120.5f};
    float cell = 11.f + 0.01f * k, want = cell;
    int n[3], m[3];
    grid_shape(lo, hi, 4200, cell, n);
    while (true) {
      for (int a = 0; a < 3; a++) m[a] = std::max(1, (int) ((hi[a] - lo[a]) / want) + 1);
      if (m[0] * m[1] * m[2] <= 4200) break;
      want *= 1.26f;
    }
    if (want != cell || m[0] != n[0] || m[1] != n[1] || m[2] != n[2]) return printf("box %d\n", k), 1;
    for (float p = lo[0] - 5; p < hi[0] + 5; p += 0.7f)
      if (grid_coord(p, lo[0], 1.f / cell, n[0]) != std::min(n[0] - 1, std::max(0, (int) ((p - lo[0]) * (1.f / cell))))) return printf("at %g\n", p), 1;
  }
  return boxes > 1000 ? 0 : 1;
}
"""


def test_every_box_fits(tmp_path):
    (tmp_path / "t.cpp").write_text(CODE)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "awsemmd_b200", "csrc"), "-o", exe, str(tmp_path / "t.cpp")],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
