"""The radices of the run-time transforms (csrc/spe_radices.h, host code,
compiled with the host compiler): at every side up to 2400 they multiply to its
smooth part, and their passes take no more shared-memory wavefronts, pass for
pass overhead included, than radices 8, 4 and the primes in that order, or than
the fewest radices, the largest first."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "spe_radices.h"
using namespace spe;

static double cost(int n, const std::vector<int>& r) {
  double w = 0;
  int ns = 1;
  for (int R : r) w += pass_wavefronts(n, ns, R) + 4.0 + 0.5 * R, ns *= R;
  return w;
}
// the fewest factors in [2, 10], the largest first
static bool fewest(int rest, int top, size_t left, std::vector<int>& r) {
  if (rest == 1) return true;
  if (left == 0) return false;
  for (int f = top; f >= 2; --f)
    if (rest % f == 0) {
      r.push_back(f);
      if (fewest(rest / f, f, left - 1, r)) return true;
      r.pop_back();
    }
  return false;
}

int main() {
  for (int n = 2; n <= 2400; ++n) {
    int smooth = 1, m = n;
    for (int f : {2, 3, 5, 7})
      for (; m % f == 0; m /= f) smooth *= f;
    int rad[kMaxRadices], prod = 1;
    const int k = choose_radices(n, smooth, rad);
    for (int i = 0; i < k; ++i) {
      if (rad[i] < 2 || rad[i] > 10) return 1;
      prod *= rad[i];
    }
    if (prod != smooth) return 2;
    const double mine = cost(n, std::vector<int>(rad, rad + k));
    std::vector<int> plain, few;
    int rest = smooth;
    for (int f : {8, 4, 2, 3, 5, 7})
      for (; rest % f == 0; rest /= f) plain.push_back(f);
    for (size_t c = 0; few.empty() && smooth > 1; ++c) fewest(smooth, 10, c, few);
    if (mine > cost(n, plain) + 1e-9 || mine > cost(n, few) + 1e-9) {
      printf("%d\n", n);
      return 3;
    }
  }
  puts("ok");
  return 0;
}
"""


def test_radices(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("needs g++")
    src, exe = tmp_path / "radices.cpp", tmp_path / "radices"
    src.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-O2", "-Wall", "-I" + os.path.join(ROOT, "s_spi_spring_gb300", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n", (r.returncode, r.stdout)
