"""Quotients and products that the FP64 kernels form with fused multiply-adds
(slbc_arith.cuh), compiled by the host compiler: the bits of plain IEEE
arithmetic over the whole range, subnormal numbers, zeros of both signs,
infinities and NaN among them.
"""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_DIR = os.path.join(ROOT, "sunlightlb_gb300", "csrc", "cuda")

HEAD = r"""
#include <cstdio>
#include <cstdint>
#include <cmath>
#include <cstring>
#include <initializer_list>
#include <limits>
#include "slbc_arith.cuh"
static uint64_t state = 88172645463325252ull;
static uint64_t bits() { state ^= state << 13; state ^= state >> 7; state ^= state << 17; return state; }
static double from(uint64_t b) { double v; std::memcpy(&v, &b, 8); return v; }
static uint64_t to(double v) { uint64_t b; std::memcpy(&b, &v, 8); return b; }
static bool same(double a, double b) { return (a != a && b != b) || to(a) == to(b); }
// a random number of exponent e (biased), any mantissa, either sign
static double number(int e) { return from((bits() & 0x800fffffffffffffull) | (uint64_t)e << 52); }
static double one_to_two() { return from((bits() & 0x000fffffffffffffull) | 1023ull << 52); }
"""

QUOTIENT = HEAD + r"""
int main() {
  const double special[] = {0.0, -0.0, std::numeric_limits<double>::infinity(), -std::numeric_limits<double>::infinity(),
                            std::nan(""), 5e-324, -5e-324, 2.2250738585072014e-308, 1.7976931348623157e308, 72.0, 1e-300};
  long wrong = 0, count = 0;
  const auto check = [&](double p, double rho, bool fast) {
    const volatile double want = p / rho;
    count++;
    bool divide = false;
    const double q = slbc::mp_quotient(p, rho, slbc::mp_reciprocal(rho), divide);
    wrong += divide ? fast : !same(q, want);
  };
  for (double p : special)
    for (double rho : special) check(p, rho, false);
  for (int e = 0; e < 2048; e++)
    for (int i = 0; i < 2000; i++) {
      check(number(e), 60.0 + 12.0 * one_to_two(), e >= 123 && e < 2047);  // densities of a flow
      check(number(e), number((int)(bits() % 2048)), false);
    }
  std::printf("%ld %ld\n", wrong, count);
}
"""

CONSTANT = HEAD + r"""
int main() {
  const double special[] = {0.0, -0.0, std::numeric_limits<double>::infinity(), -std::numeric_limits<double>::infinity(),
                            std::nan(""), 5e-324, -5e-324, 2.2250738585072014e-308, 1.7976931348623157e308};
  long wrong = 0, count = 0;
  const auto quotient = [&](double a, double b) {
    const volatile double want = a / b;
    bool divide = false;
    const double q = slbc::div_const(a, b, 1.0 / b, divide);
    count++;
    wrong += divide ? std::isfinite(a) && std::fabs(a) >= 1e-270 : !same(q, want);
  };
  const auto product = [&](double c, double p, double s) {
    const volatile double cp = c * p, want = cp + s;
    const bool rounds = slbc::scaling_rounds(c);
    count++;
    wrong += (rounds && std::fabs(c) >= 1e-300) || !same(slbc::scale_add(rounds ? slbc::rounded_scale(c, p) : c, p, s), want);
  };
  for (double a : special)
    for (double b : {72.0, 3.0}) quotient(a, b);
  for (double c : special)
    for (double s : special)
      for (double p : {0.5, 0.125}) product(c, p, s);
  for (int e = 0; e < 2047; e++)
    for (int i = 0; i < 1000; i++) {
      quotient(number(e), 72.0);
      quotient(number(e), 3.0);
      const int f = e + (int)(bits() % 121) - 60;  // an addend near c
      const double s = number(f < 0 ? 0 : f > 2046 ? 2046 : f);
      product(number(e), 0.5, s);
      product(number(e), 0.125, s);
    }
  std::printf("%ld %ld\n", wrong, count);
}
"""


def run(tmp_path, source):
    cxx = shutil.which(os.environ.get("CXX", "g++"))
    if cxx is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "arith.cpp", tmp_path / "arith"
    src.write_text(source)
    subprocess.run([cxx, "-std=c++17", "-O1", "-ffp-contract=off", "-I" + CUDA_DIR, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120).stdout
    return [int(v) for v in out.split()]


def test_tracer_quotients_equal_divisions(tmp_path):
    wrong, count = run(tmp_path, QUOTIENT)
    assert count > 8_000_000 and wrong == 0


def test_collision_quotients_and_products_equal_plain_ones(tmp_path):
    wrong, count = run(tmp_path, CONSTANT)
    assert count > 8_000_000 and wrong == 0
