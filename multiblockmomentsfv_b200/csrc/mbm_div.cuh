// mbm_div.cuh -- exact FP64 division for the bitwise kernels and the dt controller.
//
// Correctly rounded division from a shared reciprocal.
//
// Markstein's correction step (P. Markstein, "Computation of elementary functions
// on the IBM RISC System/6000 processor", IBM J. Res. Develop. 34(1):111-119, 1990;
// J.-M. Muller et al., Handbook of Floating-Point Arithmetic, 2nd ed., 2018, ch. 4):
// with r = RN(1/y) and q = RN(x*r), the remainder q*y - x is exact in one FMA and
// RN(q - (q*y - x)*r) = RN(x/y), provided x, y and the quotient stay in the normal
// range.  One reciprocal then serves every quotient with the same denominator at
// three FP64 operations each, with the same bits as IEEE x/y.  For y > 0 the negated
// remainder gives zeros their sign too: x = +-0 leaves q = +-0, the remainder q*y - x is
// +0, and -(+0)*r + q = q.  The reciprocal is Markstein's as well: the hardware
// approximation refined to within one unit in the last place (the third-order step of
// mbm_newton.cuh), then RN(r + r(1 - y r)), which is RN(1/y) unless y's significand is
// all ones (set apart).
//
// The hot path has no branch per quotient.  A set of quotients is checked together by
// integer minima and maxima of its numerators' high words (MkRange: about four integer
// instructions each, zeros admitted); a set with a numerator out of range, or whose
// denominator is not positive or out of range, is divided by IEEE division, out of line.
// Measured (bitwise step): 4 x 1024^2 cells, harmonic, 3.15 ms with a full test and a
// signed-zero select per quotient (ten integer instructions) and IEEE divisions in the
// limiter, 1.81 ms like this; 28 blocks of 30 x 10 in a stream, most sets holding a zero,
// 143 against 129 us (checking exponents alone and sorting the zeros out in a second look:
// 1.96 ms and 143 us).
// Checked against x/y, restated on the host (tests/test_exact_division.py) and on the device
// as it stands (tests/test_gpu_division.py: zeros of both signs, significands of all ones, near
// ties, the edges of the admitted range and what is outside it), and by every bitwise parity test.
#pragma once

#include <cuda_runtime.h>

#include "mbm_newton.cuh"

namespace mbm {

static __device__ __noinline__ double div_ieee(double x, double y) { return x / y; }

constexpr unsigned MK_LO = 543u << 21;             // 2^-480, as (high word << 1)
constexpr unsigned MK_SPAN = (961u << 21) - 1u;    // up to 2^481, exclusive

// The numerators of a set: in range if each is zero or has its exponent in the admitted
// range.  (high word << 1) - 1 + (low word != 0) is all ones for a zero and keeps the
// order of everything else, deep subnormals included, so its minimum finds the small ones.
struct MkRange {
  unsigned lo = ~0u, hi = 0u;
  __device__ __forceinline__ void add(double x) {
    const unsigned h = 2u * (unsigned)__double2hiint(x);
    unsigned u;
    asm("{\n .reg .u32 t;\n add.cc.u32 t, %1, 0xffffffff;\n addc.u32 %0, %2, 0xffffffff;\n}"
        : "=r"(u) : "r"(__double2loint(x)), "r"(h));
    lo = min(lo, u);
    hi = max(hi, h);
  }
  __device__ __forceinline__ bool bad() const { return lo < MK_LO || hi > MK_LO + MK_SPAN; }
};

__device__ __forceinline__ double mk_div(double x, double y, double r) {   // y > 0
  const double q = x * r;
  return fma(-fma(q, y, -x), r, q);
}

// RN(1/y) for y in range, unless y's significand is all ones
__device__ __forceinline__ double mk_rcp(double y) {
  const double r = mbm_newton::frcp(y);
  return fma(fma(-y, r, 1.0), r, r);
}
// a significand of all ones, y = 2^k (2 - 2^-52): then RN(1/y) = 2^(-k-1) (1 + 2^-52).
// Densities one rounding below 1 make this an everyday value of a stream at rho = 1.
__device__ __forceinline__ double mk_rcp_all(double y) {
  const int h = __double2hiint(y);
  const double r = mk_rcp(y);
  return ((h | (int)0xfff00000) & __double2loint(y)) == -1
             ? __hiloint2double((2045 << 20) - (h & 0x7ff00000), 1) : r;
}
// y not positive or out of range
__device__ __forceinline__ bool mk_bad_den(double y) {
  return (unsigned)__double2hiint(y) - (543u << 20) >= (961u << 20);
}

// x / y, a quotient by itself
__device__ __forceinline__ double div_rn(double x, double y) {
  MkRange g;
  g.add(x);
  const double q = mk_div(x, y, mk_rcp_all(y));
  return __builtin_expect(g.bad() || mk_bad_den(y), 0) ? div_ieee(x, y) : q;
}

}  // namespace mbm
