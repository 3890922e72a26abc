"""Row walks of the network's voxel kernels: the end of their ranges, and grids
without a voxel.

The index arithmetic (slbc_index.cuh) is compiled by the host compiler and run
at the last rows of the largest 32-bit and of a 64-bit row count, for long and
short rows: every row there is visited once, and no walk wraps.  An empty grid
is an error of the call, on the host, before any division by its sides.
"""

import os
import shutil
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_DIR = os.path.join(ROOT, "sunlightlb_gb300", "csrc", "cuda")

WALK = r"""
#include <cstdio>
#include <vector>
#include "slbc_index.cuh"
template <typename I>
int check(I rows, unsigned len) {
  const unsigned blocks = slbc::rows_grid((long long)rows, len);
  const I tail = 100000, from = rows - tail;  // the last rows, counted
  std::vector<int> seen(tail, 0);
  for (unsigned b = 0; b < blocks; b++)
    for (unsigned t = 0; t < 256; t++) {
      auto w = slbc::row_walk<I>(b, blocks, t, len);
      if (w.e != 0) continue;  // one thread per row
      if (w.row >= rows) continue;
      if (w.row < from) w.row += (from - w.row) / w.step * w.step;
      int turns = 0;
      for (I row = w.row; row < rows; row += w.step) {
        if (row >= from) seen[row - from]++;
        if (++turns > 1000000) return 1;  // wrapped
      }
    }
  for (int s : seen)
    if (s != 1) return 2;
  int n, z, y;
  slbc::row_of<I>(rows - 1, 5, 3, n, z, y);
  return ((I)n * 5 + z) * 3 + y == rows - 1 ? 0 : 3;
}
int main() {
  for (unsigned len : {1u, 2u, 7u, 255u, 256u, 1000u})
    std::printf("%d %d %d\n", check<unsigned>(0x7fffffffu, len), check<unsigned long long>((1ull << 31) + 12345, len),
                check<unsigned long long>((1ull << 32) + 7, len));
}
"""


def test_row_walks_at_their_last_rows(tmp_path):
    cxx = shutil.which(os.environ.get("CXX", "g++"))
    if cxx is None:
        pytest.skip("no C++ compiler")
    src = tmp_path / "walk.cpp"
    src.write_text(WALK)
    exe = tmp_path / "walk"
    subprocess.run([cxx, "-std=c++17", "-O1", "-I" + CUDA_DIR, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120).stdout.split()
    assert out == ["0"] * 18


EMPTY = r"""
import ctypes as C, sys
from sunlightlb_gb300 import build
d = C.CDLL(build.build())
d.slbc_last_error.restype = C.c_char_p
p, f = C.c_void_p, C.c_float
buf = p(256)  # never followed
calls = {
    "slbc_nn_pool": lambda B, D, H, W: d.slbc_nn_pool(buf, 8, 0, buf, 8, 0, B, D, H, W, 8, None),
    "slbc_nn_pool_bwd": lambda B, D, H, W: d.slbc_nn_pool_bwd(buf, 8, 0, buf, 8, 0, None, 0, 0, None, 0, 0, B, D, H, W, 8,
                                                             None),
    "slbc_nn_up": lambda B, D, H, W: d.slbc_nn_up(buf, 8, 0, buf, 8, 0, B, D, H, W, 8, None),
    "slbc_nn_up_bwd": lambda B, D, H, W: d.slbc_nn_up_bwd(buf, 8, 0, buf, 8, 0, None, 0, 0, B, D, H, W, 8, None),
    "slbc_nn_mse": lambda B, D, H, W: d.slbc_nn_mse(buf, 8, buf, 3, None, B, D, H, W, buf, 8, buf, None),
    "slbc_nn_encode": lambda B, D, H, W: d.slbc_nn_encode(buf, B, D, H, W, buf, 8, 2, None),
    "slbc_nn_decode": lambda B, D, H, W: d.slbc_nn_decode(buf, 8, buf, D if B else 0, H, W, f(1), f(0), buf, f(1), None,
                                                         None),
}
name = sys.argv[1]
for grid in ((0, 2, 2, 2), (1, 0, 2, 2), (1, 2, 0, 2), (1, 2, 2, 0), (1, 2, 2, -2)):
    assert calls[name](*grid) == 1, grid
    assert name.encode() in d.slbc_last_error() and b"empty grid" in d.slbc_last_error(), d.slbc_last_error()
"""


@pytest.mark.parametrize("name", ["slbc_nn_pool", "slbc_nn_pool_bwd", "slbc_nn_up", "slbc_nn_up_bwd", "slbc_nn_mse",
                                  "slbc_nn_encode", "slbc_nn_decode"])
def test_empty_grids_are_refused(name):
    p = subprocess.run([sys.executable, "-c", EMPTY, name], cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, (p.returncode, p.stderr[-500:])
