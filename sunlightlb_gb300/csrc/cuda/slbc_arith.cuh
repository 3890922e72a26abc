// FP64 quotients and products that kernels form with fused multiply-adds, free
// of CUDA types: the tests compile them with a host compiler and compare every
// result with plain IEEE arithmetic, bit for bit.
#ifndef SLBC_ARITH_CUH
#define SLBC_ARITH_CUH

#include <cmath>
#include <cstring>

#include "slbc_index.cuh"

namespace slbc {

SLBC_HD double fma_rn(double a, double b, double c) {
#ifdef __CUDA_ARCH__
  return __fma_rn(a, b, c);
#else
  return std::fma(a, b, c);
#endif
}

// The two words of a number, read from the bits: no FP64 operation.
struct Words {
  unsigned hi, lo;
};

SLBC_HD Words words(double v) {
#ifdef __CUDA_ARCH__
  return {(unsigned)__double2hiint(v), (unsigned)__double2loint(v)};
#else
  unsigned long long b;
  std::memcpy(&b, &v, 8);
  return {(unsigned)(b >> 32), (unsigned)b};
#endif
}

// |v| < 2^e; v infinite or NaN
SLBC_HD bool below(Words v, int e) { return (v.hi & 0x7fffffffu) < (unsigned)(1023 + e) << 20; }
SLBC_HD bool not_finite(Words v) { return (v.hi & 0x7fffffffu) >= 0x7ff00000u; }

// 1 / rho for mp_quotient; NaN, which sends it to a division, for densities
// outside [2^-64, 2^64], far from any flow's, where a quotient could leave the
// normal numbers although p is among them.
SLBC_HD double mp_reciprocal(double rho) {
  const Words w = words(rho);
  return !below(w, -64) && below(w, 64) ? 1.0 / rho : __builtin_nan("");
}

// p / rho, correctly rounded, from y = mp_reciprocal(rho): each pair of fused
// multiply-adds forms the remainder of the quotient and corrects it; after the
// first the quotient is within one ulp, so the second rounds correctly
// (Markstein).  Five FP64 operations instead of a division's ten or so.  The
// remainders must not underflow: they are multiples of 2^-105 of p, so p below
// 2^-900 (the far front of a tracer; not +0, whose quotient is right) wants a
// division, and so do infinite and undefined quotients.  `divide` is set then:
// the caller divides all its quotients again after forming them (a branch for
// each cost 10% of the FP64 update of 96^3).
SLBC_HD double mp_quotient(double p, double rho, double y, bool &divide) {
  const Words w = words(p);
  const double q0 = p * y;
  const double q1 = fma_rn(fma_rn(-rho, q0, p), y, q0);
  const double q = fma_rn(fma_rn(-rho, q1, p), y, q1);
  divide = divide || not_finite(words(q)) || (below(w, -900) && (w.hi | w.lo) != 0);
  return q;
}

// Correctly rounded a / b for a constant b with rb = RN(1/b), by Markstein's
// theorem: q = RN(a rb) is within one ulp of a / b, the remainder r = a - b q is
// exact (one fused multiply-add), and RN(q + r rb) = RN(a / b).  Three FP64
// operations instead of a full division; a = +-0 returns a (keeps the sign of
// zero).  Below 2^-900, where the remainder may underflow, and for infinities
// `divide` is set: the caller divides.
SLBC_HD double div_const(double a, double b, double rb, bool &divide) {
  const Words w = words(a);
  const bool zero = ((w.hi & 0x7fffffffu) | w.lo) == 0;
  const double q = a * rb;
  const double r = fma_rn(-q, b, a);
  const double q1 = fma_rn(r, rb, q);
  divide = divide || (!zero && below(w, -900)) || not_finite(w);
  return zero ? a : q1;
}

// c * p + s for a power of two p: where c * p is exact, one fused multiply-add
// rounds like the multiplication and the addition.  For p = 1/2 or 1/8 that is
// so unless c * p is subnormal: for such c (zero apart) scaling_rounds is true,
// and c = rounded_scale(c, p) makes the two agree again (c * p rounded, which
// the division by p keeps).
SLBC_HD double scale_add(double c, double p, double s) { return fma_rn(c, p, s); }
SLBC_HD bool scaling_rounds(double c) {
  const Words w = words(c);
  return below(w, -1000) && ((w.hi & 0x7fffffffu) | w.lo) != 0;
}
SLBC_HD double rounded_scale(double c, double p) { return c * p * (1.0 / p); }

}  // namespace slbc

#endif
