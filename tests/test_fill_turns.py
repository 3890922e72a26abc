"""Tracer fills over several turns of the grid, and the index arithmetic of
their loop at the largest lattice.

A field of more nodes than the grid has threads, every kind of region, against
numpy (values exact in FP32, so equal bits; the injected total to the rounding
of 4e5 FP64 additions of O(1) terms, 4e5 x 2^-53 x 4e5 = 2e-5 at most, here
asked to 1e-9).  A region of an unknown kind holds no node.  The loop itself,
grid_turns, is compiled by the host compiler and run over 2^31 - 1 elements.
"""

import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_DIR = os.path.join(ROOT, "sunlightlb_gb300", "csrc", "cuda")

TURNS = r"""
#include <cstdio>
#include "slbc_index.cuh"
int main() {
  const unsigned count = 0x7fffffffu, step = 608u * 256u, firsts[3] = {0u, 1u, step - 1u};
  for (unsigned first : firsts) {
    unsigned turns = 0, last = 0;
    bool inside = true;
    slbc::grid_turns(first, step, count, [&](unsigned e) {
      inside = inside && e < count && (turns == 0 || e - last == step);
      last = e;
      turns++;
    });
    std::printf("%d %u %u\n", inside ? 1 : 0, turns, (count - first + step - 1u) / step);
  }
}
"""


def test_grid_turns_at_the_largest_lattice(tmp_path):
    cxx = shutil.which(os.environ.get("CXX", "g++"))
    if cxx is None:
        pytest.skip("no C++ compiler")
    src = tmp_path / "turns.cpp"
    src.write_text(TURNS)
    exe = tmp_path / "turns"
    subprocess.run([cxx, "-std=c++17", "-O1", "-I" + CUDA_DIR, str(src), "-o", str(exe)], check=True)
    for line in subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60).stdout.splitlines():
        inside, turns, want = map(int, line.split())
        assert inside == 1 and turns == want


DIMS = (70, 75, 80)  # 420,000 nodes: three turns of 608 blocks of 256
REGIONS = [  # kind, geo
    (0, ()),
    (1, (3.0, 60.0, 1.0, 70.0, 2.0, 77.0)),
    (2, (0, 69)), (2, (1, 74)), (2, (2, 79)),
    (3, (30.5, 35.0, 37.0, 40.0)),
    (4, (2, 0, 30.5, 35.0, 37.0)), (4, (0, 1, 30.5, 35.0, 37.0)),
    (5, (1.0,) * 6), (-1, (1.0,) * 6),
]


def region(kind, geo):
    i, j, k = np.meshgrid(*(np.arange(n, dtype=float) for n in DIMS), indexing="ij")
    if kind == 0:
        return np.ones(DIMS, bool)
    if kind == 1:
        return ((i > geo[0]) & (i < geo[1]) & (j > geo[2]) & (j < geo[3]) & (k > geo[4]) & (k < geo[5]))
    if kind == 2:
        return (i, j, k)[geo[0]] == geo[1]
    if kind == 3:
        return (i - geo[1]) ** 2 + (j - geo[2]) ** 2 + (k - geo[3]) ** 2 < geo[0] ** 2
    if kind == 4:
        u, w = (j, k) if geo[0] == 0 else (i, j) if geo[0] == 2 else (i, k)
        inside = (u - geo[3]) ** 2 + (w - geo[4]) ** 2 < geo[2] ** 2
        return ~inside if geo[1] else inside
    return np.zeros(DIMS, bool)


@pytest.mark.gpu
@pytest.mark.parametrize("f64", [1, 0])
@pytest.mark.parametrize("kind, geo", REGIONS)
def test_fills_of_several_turns(gpu, kind, geo, f64):
    d, n = gpu.dll, int(np.prod(DIMS))
    h, t = C.c_void_p(), C.c_void_p()
    assert d.slbc_create(C.byref(h), *DIMS, 0) == 0
    assert d.slbc_mp_create(h, C.byref(t), f64) == 0
    old = np.random.default_rng(kind + 7).integers(0, 64, n) / 16.0
    got, total = np.empty(n), C.c_double()
    assert d.slbc_mp_put(t, old.ctypes.data_as(C.c_void_p)) == 0
    arr = (C.c_double * 6)(*geo)
    assert d.slbc_mp_fill(t, kind, arr, C.c_double(0.5)) == 0
    assert d.slbc_mp_get(t, got.ctypes.data_as(C.c_void_p)) == 0
    assert d.slbc_mp_injected(t, 1, C.byref(total)) == 0
    d.slbc_mp_destroy(t)
    d.slbc_destroy(h)
    inside = region(kind, geo).ravel()
    assert np.array_equal(got, np.where(inside, 0.5, old))
    assert abs(total.value - (0.5 - old[inside]).sum()) <= 1e-9 * max(1.0, np.abs(old).sum())
