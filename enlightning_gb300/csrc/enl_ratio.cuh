// The ratio test of the hybrid switch (rhs_hybrid_high_llf.m4:239-256) and of
// tag_cells (tag_cells.m4:58-108), decided bit for bit as the reference's
// division decides it.
//
// (2 |t1 t2| + ep) / (t1^2 + t2^2 + ep) < 0.9999 with t1, t2 differences of
// neighbouring values.  FP64 operations are what these tests cost (the pipe
// does 2 per SM and clock), so the ratio is first formed in single precision
// from the differences' exponents and leading 20 mantissa bits: within 4e-6 of
// the exact one, it decides unless it lies within 1e-5 of the threshold.  What
// is left is estimated in FP64 as num * rcp64(den), within 2^-50, and divided
// only within 2^-44 of the threshold.  Per cell that is 8 FP64 operations in
// place of about 70 for the switch.
#pragma once
#include "enl_rcp.cuh"

namespace enl {

// ep for the single-precision test; 0 where ep is outside the range in which
// neither ep nor a product of differences can leave single precision (the
// test then goes to FP64 at once).
inline float ratio_eps32(double ep) { return ep >= 0x1p-60 && ep <= 0x1p60 ? (float)ep : 0.f; }

// Single-precision value of a double's magnitude from its high word, truncated
// to 20 mantissa bits; below 2^-100 (its square then vanishes beside ep) 0.
__device__ __forceinline__ float ratio_mag32(unsigned a) {
  return a >= ((1023u - 100u) << 20) ? __uint_as_float((a - (896u << 20)) << 3) : 0.f;
}

// In FP64.  Two zero differences give the ratio ep / ep, 1 or NaN: not below.
// For ep above 2^-1000 numerator and denominator are normal and positive, and
// a positive quotient (or NaN, whose pattern is above the threshold's) orders
// as its bit pattern.
static __device__ __noinline__ bool ratio_below_exact(double t1, double t2, double ep) {
  constexpr double kLo = Lit::c0_9999 * (1.0 - 0x1p-44);
  constexpr double kHi = Lit::c0_9999 * (1.0 + 0x1p-44);
  const unsigned long long mag =
      ((unsigned long long)__double_as_longlong(t1) | (unsigned long long)__double_as_longlong(t2)) << 1;
  if (mag == 0ull) return false;
  const double num = __dadd_rn(__dmul_rn(2.0, fabs(__dmul_rn(t1, t2))), ep);
  const double den = __dadd_rn(__dadd_rn(__dmul_rn(t1, t1), __dmul_rn(t2, t2)), ep);
  if (!(ep > 0x1p-1000)) return __ddiv_rn(num, den) < Lit::c0_9999;
  const unsigned long long qb = (unsigned long long)__double_as_longlong(num * rcp64(den));
  if (qb < (unsigned long long)__double_as_longlong(kLo)) return true;
  return qb <= (unsigned long long)__double_as_longlong(kHi) && __ddiv_rn(num, den) < Lit::c0_9999;
}

__device__ __forceinline__ bool ratio_below(double t1, double t2, double ep, float ep32) {
  const unsigned a = (unsigned)__double2hiint(t1) & 0x7fffffffu, b = (unsigned)__double2hiint(t2) & 0x7fffffffu;
  if (ep32 > 0.f && max(a, b) < ((1023u + 50u) << 20)) {
    const float x = ratio_mag32(a), y = ratio_mag32(b);
    const float num = fmaf(2.0f * x, y, ep32), den = fmaf(x, x, fmaf(y, y, ep32));
    if (num > 0.99991f * den) return false;
    if (num < 0.99989f * den) return true;
  }
  return ratio_below_exact(t1, t2, ep);
}

// The switch along one direction: r[0..4] = rho at offsets -2..2; 1 if any of
// the ratios at offsets -1, 0, 1 is below the threshold.
__device__ __forceinline__ int sensor_line(const double r[5], double ep, float ep32) {
  double t[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) t[q] = __dsub_rn(r[q + 1], r[q]);
  return ratio_below(t[0], t[1], ep, ep32) || ratio_below(t[1], t[2], ep, ep32) || ratio_below(t[2], t[3], ep, ep32);
}

// The four tests of tag_cells at a cell of row pitch `pitch`: the source, then
// the density.  Three values with the same bits are never below the threshold
// (the ratio is ep/ep = 1 or NaN), whatever ep is: where a field is at rest,
// which is most of a level, no FP64 operation is left.  (Eight subtractions a
// cell were 136 us of a 4096 x 2048 level's tags, 69 without; FP32 storage 70 and 46.)
__device__ __forceinline__ bool tag_line64(double m, double c, double p, double ep, float epf) {
  const long long b = __double_as_longlong(c);
  if (__double_as_longlong(m) == b && __double_as_longlong(p) == b) return false;
  return ratio_below(__dsub_rn(c, m), __dsub_rn(p, c), ep, epf);
}
__device__ __forceinline__ bool tag_cell64(const double* H, const double* W, long pitch, double ep0, float ep0f,
                                           double ep1, float ep1f) {
  const double h[5] = {H[0], H[-1], H[1], H[-pitch], H[pitch]};
  const double r[5] = {W[0], W[-1], W[1], W[-pitch], W[pitch]};
  return tag_line64(h[1], h[0], h[2], ep0, ep0f) || tag_line64(h[3], h[0], h[4], ep0, ep0f) ||
         tag_line64(r[1], r[0], r[2], ep1, ep1f) || tag_line64(r[3], r[0], r[4], ep1, ep1f);
}

}  // namespace enl
