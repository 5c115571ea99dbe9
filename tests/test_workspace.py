"""The crossover's workspace (csrc/spe_workspace.h, host code, compiled with
the host compiler): for populations far larger than a test can run, with and
without the average, every array has the size its kernels index and lies inside
the bytes that are asked for, and a workspace that is one byte short is
refused."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cstdint>
#include <utility>
#include <vector>
#include "spe_workspace.h"
using namespace spe_detail;
using spe::CrossChild;
using spe::ShiftItem;

int main() {
  for (size_t P : {1, 6, 224, 225, 256, 448, 512, 1024, 4096})
    for (int pairs : {3, 4})
      for (size_t n : {63, 64, 512}) {
        const int per = pairs + 1;
        const size_t npix = n * n, nred = 4 * (n / 8 + 1), maps = 20 * P;
        const size_t bytes = CrossWork::bytes(P, npix, nred, pairs, per, maps);
        char* base = reinterpret_cast<char*>(size_t(1) << 20);  // never dereferenced
        Carve cv{base, bytes};
        const CrossWork w(cv, P, npix, nred, pairs, per, maps);
        if (!cv.fits()) return 1;
        Carve cut{base, bytes - 1};
        const CrossWork v(cut, P, npix, nred, pairs, per, maps);
        (void)v;
        if (cut.fits()) return 2;
        // (start, bytes that are written) in the order of the addresses
        const std::vector<std::pair<const void*, size_t>> a = {
            {w.D, (P + 1) * npix * 8}, {w.scratch, P * pairs * npix * 8}, {w.W, P * per * npix * 8},
            {w.C, P * npix * 8}, {w.Ws, 3 * P * npix * 4}, {w.part, P * pairs * nred * 8},
            {w.part2, P * pairs * nred * 8}, {w.psum, (P + 1) * nred * 8}, {w.peaks, P * pairs * 32},
            {w.sums, (P + 1) * 16}, {w.xi, P * pairs * 4}, {w.ri, P * pairs * 4},
            {w.items, P * per * sizeof(ShiftItem)}, {w.children, P * sizeof(CrossChild)}, {w.bits, P * npix / 4},
            {w.cmaps, maps * 4}};
        size_t end = size_t(1) << 20;
        for (const auto& r : a) {
          const size_t at = reinterpret_cast<size_t>(r.first);
          if (at < end || at % 256) return 3;
          end = at + r.second;
        }
        if (end > (size_t(1) << 20) + bytes) return 4;
        if (P * per < P * size_t(pairs)) return 5;  // W: scratch of the second product
      }
  puts("ok");
  return 0;
}
"""


def test_crossover_workspace(tmp_path):
    gxx, cuda = shutil.which("g++"), "/usr/local/cuda/include"
    if not gxx or not os.path.isdir(cuda):
        pytest.skip("needs g++ and the CUDA headers")
    src, exe = tmp_path / "workspace.cpp", tmp_path / "workspace"
    src.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-Wall", "-I" + os.path.join(ROOT, "s_spi_spring_gb300", "csrc"), "-I" + cuda,
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n", (r.returncode, r.stdout)
