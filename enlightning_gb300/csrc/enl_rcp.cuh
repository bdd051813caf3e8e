// Seeded FP64 reciprocal.
#pragma once
#include "enl_common.cuh"

namespace enl {

// Single-precision reciprocal of the hardware (rcp.approx, within 1 ulp).
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Reciprocal of a double.  For positive normal x within the float exponent
// range, the double's exponent and top 20 mantissa bits are moved into a
// float by integer operations, the hardware single-precision reciprocal gives
// a seed r with |1 - x r| < 2^-19, and one Newton step with its cubic term,
// r (1 + e + e^2) with e = 1 - x r, leaves |1 - x r'| = |e|^3 < 2^-57, below
// FP64 rounding.  Zero, negative, non-finite and out-of-range arguments take
// the division.  All bit manipulation is on unsigned integers, so no shift
// overflows.
__device__ __forceinline__ double rcp64(double x) {
  const unsigned hi = (unsigned)__double2hiint(x);
  const unsigned e = hi >> 20;  // sign and biased exponent
  if (e - (1023u - 125u) > 250u) return 1.0 / x;
  const float xf = __uint_as_float((hi - ((1023u - 127u) << 20)) << 3);
  const unsigned rb = __float_as_uint(rcp_approx(xf));
  const double r = __hiloint2double((int)((rb >> 3) + ((1023u - 127u) << 20)), (int)(rb << 29));
  const double ee = fma(-x, r, 1.0);
  return fma(r, fma(ee, ee, ee), r);
}

}  // namespace enl
