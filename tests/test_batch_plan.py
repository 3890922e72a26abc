"""How a batch is cut into sets (slbc_sets.cuh, compiled by the host compiler):
every member in one set, sets of the L2's size however unequal the members, no
small set left over, and few launch classes per set.
"""

import os
import random
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_DIR = os.path.join(ROOT, "sunlightlb_gb300", "csrc", "cuda")
MB = 1 << 20
WHOLE, SET = 112 * MB, 64 * MB

MAIN = r"""
#include <cstdio>
#include "slbc_sets.cuh"
int main() {
  int n;
  while (std::scanf("%d", &n) == 1) {
    std::vector<long long> bytes(n);
    std::vector<int> cls(n);
    for (int d = 0; d < n; d++) if (std::scanf("%lld %d", &bytes[d], &cls[d]) != 2) return 1;
    for (const auto &set : slbc::batch_sets(bytes, cls)) {
      for (int d : set) std::printf("%d ", d);
      std::printf("; ");
    }
    std::printf("\n");
  }
}
"""


@pytest.fixture(scope="module")
def cut(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("sets")
    (d / "m.cpp").write_text(MAIN)
    subprocess.run([cxx, "-O1", "-std=c++17", "-x", "c++", "-I" + CUDA_DIR, str(d / "m.cpp"), "-o", str(d / "m")], check=True)

    def run(bytes_, cls=None):
        cls = cls or [0] * len(bytes_)
        text = f"{len(bytes_)} " + " ".join(f"{b} {c}" for b, c in zip(bytes_, cls))
        out = subprocess.run([str(d / "m")], input=text, capture_output=True, text=True, check=True).stdout
        return [[int(v) for v in s.split()] for s in out.split(";") if s.strip()]

    return run


def fp32(side):
    return side ** 3 * 62


def check(sets, bytes_):
    assert sorted(d for s in sets for d in s) == list(range(len(bytes_)))
    total = sum(bytes_)
    if total <= WHOLE:
        assert len(sets) <= 1
        return
    for s in sets:
        b = sum(bytes_[d] for d in s)
        big = [d for d in s if bytes_[d] > SET]
        assert len(big) <= 1
        if big:
            # others only beside a member that does not fit the L2 by itself, or where all fit
            assert len(s) == 1 or bytes_[big[0]] > WHOLE or b <= WHOLE
        else:
            # at most a share of kBatchSet and half a member, and a small rest
            assert b <= SET + max(bytes_[d] for d in s) // 2 or b <= WHOLE
    small = [s for s in sets if sum(bytes_[d] for d in s) < SET // 4]
    rest = sum(b for b in bytes_ if b <= SET)
    assert len(small) <= (1 if rest < SET // 2 else 0), sets


def test_one_large_member_among_small_ones(cut):
    for large, small, count in ((288, 24, 64), (256, 48, 40), (512, 24, 64), (128, 24, 300)):
        for bytes_ in ([fp32(large)] + [fp32(small)] * count, [fp32(small)] * count + [fp32(large)],
                       [fp32(small)] * (count // 2) + [fp32(large)] + [fp32(small)] * (count - count // 2)):
            sets = cut(bytes_)
            check(sets, bytes_)
            rest = fp32(small) * count
            assert len(sets) <= 1 + -(-rest // SET), (large, small, len(sets))


def test_equal_members_keep_equal_sets(cut):
    bytes_ = [fp32(24 + (i * 40) // 63) for i in range(64)]
    sets = cut(bytes_)
    check(sets, bytes_)
    assert len(sets) == -(-sum(bytes_) // SET)
    assert cut([fp32(48)] * 16) == [list(range(16))]  # 110 MB: one set
    assert cut([]) == []


def test_members_go_class_by_class(cut):
    bytes_, cls = [fp32(48)] * 64, [i % 8 for i in range(64)]
    sets = cut(bytes_, cls)
    check(sets, bytes_)
    assert max(len({cls[d] for d in s}) for s in sets) <= 2


def test_any_members(cut):
    rng = random.Random(3)
    for _ in range(400):
        n = rng.randint(1, 60)
        kind = rng.randrange(3)
        sides = [rng.choice((16, 24, 200, 300)) if kind == 0 else int(2 ** rng.uniform(3, 8.3)) if kind == 1
                 else rng.randint(60, 100) for _ in range(n)]
        bytes_ = [fp32(s) for s in sides]
        check(cut(bytes_, [rng.randrange(8) for _ in range(n)]), bytes_)
