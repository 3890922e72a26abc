"""The march of tracer blocks (march_planes, compiled by the host compiler) is
the best of all counts of blocks, and its search stays short on long lattices.
"""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_DIR = os.path.join(ROOT, "sunlightlb_gb300", "csrc", "cuda")

MAIN = r"""
#include <chrono>
#include <initializer_list>
#include <cstdio>
#include "slbc_index.cuh"
int all(int esi, long long tiles, long long slots, int most = 1 << 30, int halo = 2, int tail = 0) {
  long long best = 0;
  int planes = 1;
  for (int chunks = 1; chunks <= esi; chunks++) {
    const int p = (esi + chunks - 1) / chunks;
    if (p > most) continue;
    const long long waves = (tiles * ((esi + p - 1) / p) + slots - 1) / slots, cost = (6 * waves + tail) * (p + halo);
    if (best == 0 || cost < best || (tail && cost == best)) { best = cost; planes = p; }
  }
  return planes;
}
int main() {
  int wrong = 0;
  for (int esi = 1; esi < 700; esi++)
    for (long long tiles : {1, 2, 7, 36, 100, 512, 9999})
      for (int b : {2, 3, 4}) {
        wrong += all(esi, tiles, 152 * b) != slbc::march_planes(esi, tiles, 152 * b);
        wrong += all(esi, tiles, 152 * b, 4) != slbc::march_planes(esi, tiles, 152 * b, 4);
        wrong += slbc::march_planes(esi, tiles, 152 * b, 4) > 4;
        wrong += all(esi, tiles, 152 * b, 1 << 30, 1, 12) != slbc::march_planes(esi, tiles, 152 * b, 1 << 30, 1, 12);
        wrong += all(esi, tiles, 152 * b, 1 << 30, 2, 1) != slbc::march_planes(esi, tiles, 152 * b, 1 << 30, 2, 1);
      }
  for (int esi : {4096, 10007, 65535})
    for (long long tiles : {1, 3, 40}) wrong += all(esi, tiles, 456) != slbc::march_planes(esi, tiles, 456);
  const auto time = [](auto f) {
    const auto t0 = std::chrono::steady_clock::now();
    int sum = 0;
    for (int r = 0; r < 20; r++) sum += f(65535 - r, 2, 456, 1 << 30, 2, 0);
    const std::chrono::duration<double, std::micro> d = std::chrono::steady_clock::now() - t0;
    return sum > 0 ? d.count() / 20 : -1.0;
  };
  std::printf("%d %.2f %.2f\n", wrong, time(all), time(slbc::march_planes));
}
"""


def test_march(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    (tmp_path / "m.cpp").write_text(MAIN)
    subprocess.run([cxx, "-O2", "-std=c++17", "-x", "c++", "-I" + CUDA_DIR, str(tmp_path / "m.cpp"), "-o", str(tmp_path / "m")],
                   check=True)
    wrong, before, now = subprocess.run([str(tmp_path / "m")], check=True, capture_output=True, text=True).stdout.split()
    assert wrong == "0"
    assert float(now) < 0.1 * float(before)  # some 500 candidates of 65,535
    print(before, now)
