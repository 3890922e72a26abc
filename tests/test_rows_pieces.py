"""Row walks of the network's voxel kernels on grids of few long rows: rows are cut
into pieces for enough blocks, and every element has its one turn (slbc_index.cuh,
run by the host compiler).  The kernels on such grids are in test_gpu_glue_long.py.
"""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_DIR = os.path.join(ROOT, "sunlightlb_gb300", "csrc", "cuda")

MAIN = r"""
#include <cstdio>
#include <initializer_list>
#include <vector>
#include "slbc_index.cuh"
template <typename I>
int check(I rows, unsigned len) {
  const unsigned blocks = slbc::rows_grid((long long)rows, len);
  std::vector<unsigned char> seen((size_t)rows * len, 0);
  unsigned busy = 0, longest = 0;
  for (unsigned b = 0; b < blocks; b++) {
    bool any = false;
    for (unsigned t = 0; t < 256; t++) {
      const auto w = slbc::row_turns<I>(b, blocks, t, rows, len);
      unsigned mine = 0;
      for (I turn = w.first; turn < w.turns; turn += w.step) {
        const auto p = w.piece(turn);
        if (p.row >= rows || p.end > len) return 1;
        for (unsigned e = p.e; e < p.end; e += 256, mine++) seen[(size_t)p.row * len + e]++;
      }
      any = any || mine;
      longest = mine > longest ? mine : longest;
    }
    busy += any;
  }
  for (unsigned char s : seen)
    if (s != 1) return 2;
  // no thread has far more than its share of a full GPU, or of blocks of two turns
  const double share = (double)rows * len / (256.0 * slbc::kRowBlocks);
  if (longest > 2 * share + 2) return 3;
  return busy == blocks ? 0 : 4;
}
int main() {
  for (unsigned rows : {1u, 2u, 3u, 4u, 7u, 24u, 100u, 607u, 1216u, 2431u, 2432u, 2433u, 5000u})
    for (unsigned len : {1u, 5u, 64u, 255u, 256u, 257u, 511u, 512u, 513u, 1000u, 1024u, 4095u, 20000u})
      if ((double)rows * len < 3e7)
        if (const int rc = check<unsigned>(rows, len) * 10 + check<unsigned long long>(rows, len))
          std::printf("%u rows of %u: %d\n", rows, len, rc);
  for (unsigned len : {100003u, 640000u, 5120000u, 20000000u})
    if (const int rc = check<unsigned>(1u, len)) std::printf("1 row of %u: %d\n", len, rc);
}
"""


def test_pieces(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    (tmp_path / "m.cpp").write_text(MAIN)
    subprocess.run([cxx, "-O2", "-std=c++17", "-x", "c++", "-I" + CUDA_DIR, str(tmp_path / "m.cpp"), "-o", str(tmp_path / "m")],
                   check=True)
    out = subprocess.run([str(tmp_path / "m")], check=True, capture_output=True, text=True, timeout=600).stdout
    assert out == ""
