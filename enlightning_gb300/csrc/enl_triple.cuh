// WENO flux differences in triple-single arithmetic.
//
// A WENO5 cell needs 40 reconstructions (5 fields, 2 directions, 2 signs, 2
// faces), each with three smoothness indicators and a normalised weighted sum.
// In FP64 they are what the right-hand side spends its time on: the FP64 pipe
// completes 2 fused multiply-adds per SM and clock, the FP32 pipe 128.  Here
// the nonlinear part runs on the FP32 pipe with numbers of three floats
// (value = h + m + l, each word about 2^-23 of the one before, relative error
// of one operation below 2^-60).  One flux difference (four reconstructions)
// took about 26 clocks of an SM; in FP64 it was about 155 instructions of the
// FP64 pipe, 78 clocks.  On the Mach shock (1024x512, two levels, WENO nearly
// everywhere) an FP64 step went from 29.8 to 11.3 ms, on the three-level line
// source with its host exchange from 9.2 to 5.0 ms.  (Since then t3_grid has
// taken a tenth off its operations.)
//
// Accuracy, against 128-bit arithmetic on 200,000 random stencils each (error
// over the stencil's largest split flux, RMS): smooth waves 2.0e-18 (FP64
// routine 2.4e-16), 1 % density noise 2.4e-18 (2.8e-16), a density jump of
// 1.8 4.9e-17 (2.2e-16), white noise 1.1e-16 (1.8e-16).  What is left is the
// rounding of the FP64 differences.
//
// The building blocks are the error-free transformations of Knuth (two-sum)
// and Dekker/Veltkamp with a fused multiply-add (two-product), and a Newton
// reciprocal.  Both signs of the split flux run through the same code on
// packed float pairs (fma.rn.f32x2 and friends: half the issue slots; 26
// clocks per flux difference against 32 in scalar form).
//
// Algebra.  With the split fluxes x_i = F_i/2 + a/2 w_i and m_i = F_i/2 -
// a/2 w_i at offsets i - 3 (i = 0..6) and y_j = m_{6-j}, the reconstructions
// of rhs_hybrid_high_llf.m4:286-358 are mirror images: wenom(a,b,c,d,e) =
// wenop(e,d,c,b,a), so the flux difference is R(x) - R(y) with R the
// difference of the two wenop values on x_0..x_4 and x_1..x_5.  Every
// candidate polynomial is the middle one plus a multiple of a third
// difference, so with the differences d_j = x_{j+1} - x_j, t_j = d_{j+1} -
// d_j and D_j = t_{j+1} - t_j
//   6 wenop(lo) = f1 - w0 D_1 - 2 w2 D_0,
// and R needs nothing but differences.  The routine therefore takes the
// differences of F/2 and w in FP64 (F/2 is a rounded half flux, and a
// difference is rounded unless the two lie within a factor of two of each
// other), forms d_j for both signs (10 fused multiply-adds, rounded) and
// converts those to three words, scaled by the largest one's power of two, so
// that no value of the state overflows or underflows the single-precision
// range: exactly, down to 2^-75 of the largest.
#pragma once
#include "enl_rcp.cuh"

namespace enl {

// Two floats in one 64-bit register: .x belongs to x (the plus sign), .y to y.
typedef unsigned long long f2;
__device__ __forceinline__ f2 f2_pack(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void f2_unpack(f2 v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f2 f2_both(float c) { return f2_pack(c, c); }
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2 f2_neg(f2 a) {
  float x, y;
  f2_unpack(a, x, y);
  return f2_pack(-x, -y);
}
__device__ __forceinline__ f2 f2_sub(f2 a, f2 b) { return f2_fma(b, f2_both(-1.f), a); }

// s + e = a + b exactly.
__device__ __forceinline__ void f2_two_sum(f2 a, f2 b, f2& s, f2& e) {
  s = f2_add(a, b);
  const f2 z = f2_sub(s, a);
  e = f2_add(f2_sub(a, f2_sub(s, z)), f2_sub(b, z));
}
// s + e = a + c b exactly, c a power of two of either sign.
__device__ __forceinline__ void f2_two_sum_c(f2 a, float c, f2 b, f2& s, f2& e) {
  if (c == 1.f) return f2_two_sum(a, b, s, e);
  s = f2_fma(b, f2_both(c), a);
  const f2 z = f2_sub(s, a);
  e = f2_add(f2_sub(a, f2_sub(s, z)), f2_fma(b, f2_both(c), f2_neg(z)));
}

struct T3 {
  f2 h, m, l;
};

// a + c b, c a power of two of either sign (a constant at the call).
__device__ __forceinline__ T3 t3_add(T3 a, float c, T3 b) {
  f2 s, e, s1, e1, m, e2;
  f2_two_sum_c(a.h, c, b.h, s, e);
  f2_two_sum_c(a.m, c, b.m, s1, e1);
  f2_two_sum(s1, e, m, e2);
  return T3{s, m, f2_add(f2_add(f2_fma(b.l, f2_both(c), a.l), e1), e2)};
}
__device__ __forceinline__ T3 t3_add_f(T3 a, f2 c) {
  f2 s, e, m, e2;
  f2_two_sum(a.h, c, s, e);
  f2_two_sum(a.m, e, m, e2);
  return T3{s, m, f2_add(a.l, e2)};
}
__device__ __forceinline__ T3 t3_sqr(T3 a) {
  const f2 p = f2_mul(a.h, a.h), e = f2_fma(a.h, a.h, f2_neg(p));
  const f2 t = f2_add(a.h, a.h), q = f2_mul(t, a.m), f = f2_fma(t, a.m, f2_neg(q));
  f2 s, r;
  f2_two_sum(q, e, s, r);
  return T3{p, s, f2_fma(a.m, a.m, f2_fma(t, a.l, f2_add(f, r)))};
}
__device__ __forceinline__ T3 t3_mul(T3 a, T3 b) {
  const f2 p = f2_mul(a.h, b.h), e = f2_fma(a.h, b.h, f2_neg(p));
  const f2 q1 = f2_mul(a.h, b.m), f1 = f2_fma(a.h, b.m, f2_neg(q1));
  const f2 q2 = f2_mul(a.m, b.h), g2 = f2_fma(a.m, b.h, f2_neg(q2));
  f2 s1, r1, s2, r2;
  f2_two_sum(q1, q2, s1, r1);
  f2_two_sum(s1, e, s2, r2);
  return T3{p, s2,
            f2_fma(a.m, b.m, f2_fma(a.h, b.l, f2_fma(a.l, b.h, f2_add(f2_add(f1, g2), f2_add(r1, r2)))))};
}
__device__ __forceinline__ T3 t3_mul_f(T3 a, f2 c) {
  const f2 p = f2_mul(c, a.h), e = f2_fma(c, a.h, f2_neg(p));
  const f2 q = f2_mul(c, a.m), f = f2_fma(c, a.m, f2_neg(q));
  f2 s, r;
  f2_two_sum(q, e, s, r);
  return T3{p, s, f2_fma(c, a.l, f2_add(f, r))};
}

// Sums of the differences with small whole coefficients, on a common grid: the
// words of a value below 2 in magnitude are put on multiples of 2^-19 and
// 2^-40 and a rest (12 operations), where values of the same scale add word
// by word, exactly in the first two (up to 8 of them: 2^24 steps of the grid),
// three operations a sum; what is then squared is made three words of
// decreasing size again (nine).  Against t3_add, 22 operations, 15 times a flux
// difference, it leaves 195 of 330 (of 1331 in all): the Mach shock's step
// 9.55 -> 9.00 ms, the line source's 3.26 -> 3.11, a small two-level run's 0.364
// -> 0.344.  The grid ends near 2^-63 of the largest
// difference: a small value next to a large one loses relative accuracy, but
// the weights it forms differ from 0 and 1 only where the differences they
// multiply are as small (errors on 200,000 random stencils as in the heading;
// noise of 1e-11 beside a jump 2.0e-20 of the flux instead of 1.3e-21).
__device__ __forceinline__ T3 t3_grid(T3 a) {
  const f2 C1 = f2_both(24.f), C2 = f2_both(0x1.8p-17f);  // units in the last place 2^-19, 2^-40
  const f2 H = f2_sub(f2_add(a.h, C1), C1), r = f2_sub(a.h, H);
  const f2 s = f2_add(C2, r), s2 = f2_add(s, a.m);
  return T3{H, f2_sub(s2, C2), f2_add(f2_add(f2_sub(r, f2_sub(s, C2)), f2_sub(a.m, f2_sub(s2, s))), a.l)};
}
// a + c b on the grid.
__device__ __forceinline__ T3 t3_lin(T3 a, float c, T3 b) {
  if (c == 1.f) return T3{f2_add(a.h, b.h), f2_add(a.m, b.m), f2_add(a.l, b.l)};
  const f2 k = f2_both(c);
  return T3{f2_fma(b.h, k, a.h), f2_fma(b.m, k, a.m), f2_fma(b.l, k, a.l)};
}
__device__ __forceinline__ T3 t3_norm(T3 a) {
  const f2 u = f2_add(a.m, a.l), v = f2_sub(a.l, f2_sub(u, a.m));
  const f2 s = f2_add(a.h, u), e = f2_sub(u, f2_sub(s, a.h)), m = f2_add(e, v);
  return T3{s, m, f2_sub(v, f2_sub(m, e))};
}

// K / q for q > 0 normal, K a power of two.  One Newton step makes the
// hardware seed y accurate to half a unit, so that the residual 1 - q.h y is
// exact; then 1 / q = y (1 + r + r^2) with r = 1 - q y, |r| < 2^-21, whose
// next term is below 2^-63.
__device__ __forceinline__ T3 t3_rcp(T3 q, f2 K) {
  float a, b;
  f2_unpack(q.h, a, b);
  const f2 nq = f2_neg(q.h), nm = f2_neg(q.m), one = f2_both(1.f);
  f2 y = f2_pack(rcp_approx(a), rcp_approx(b));
  y = f2_fma(y, f2_fma(nq, y, one), y);
  const f2 r = f2_fma(nq, y, one), p = f2_mul(nm, y), ep = f2_fma(nm, y, f2_neg(p));
  f2 rs, re;
  f2_two_sum(r, p, rs, re);
  re = f2_add(re, f2_fma(f2_neg(q.l), y, ep));
  const f2 yk = f2_mul(y, K), m = f2_mul(yk, rs), em = f2_fma(yk, rs, f2_neg(m));
  return T3{yk, m, f2_fma(yk, f2_fma(rs, rs, re), em)};
}

// Power of two of the smallest of three positive floats per half: weights are
// formed from K / q, at most 2 for the smallest q, so the largest weight is
// of order 1 and those that underflow are below 2^-126 of it.
__device__ __forceinline__ float pow2_of(float a) { return __uint_as_float(__float_as_uint(a) & 0x7f800000u); }
__device__ __forceinline__ f2 f2_pow2_min(f2 a, f2 b) {
  float ax, ay, bx, by;
  f2_unpack(a, ax, ay);
  f2_unpack(b, bx, by);
  return f2_pack(pow2_of(fminf(ax, bx)), pow2_of(fminf(ay, by)));
}
__device__ __forceinline__ f2 f2_pow2_min(f2 a, f2 b, f2 c) { return f2_pow2_min(f2_pow2_min(a, b), f2_pow2_min(c, c)); }

// Exact conversion of a double times 2^(127 - E) (E the biased exponent given
// as bias20 = (E - 127) << 20): 24 + 23 + 6 bits of its mantissa.  Values
// below 2^-75 of 2^(E - 1023) become 0.
__device__ __forceinline__ void t3_split(double x, int bias20, float& h, float& m, float& l) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const int t = (int)(hi & 0x7fffffffu) - bias20;
  const unsigned f = ((unsigned)t << 3) | (lo >> 29) | (hi & 0x80000000u);
  const unsigned b1 = (f & 0xff800000u) - (23u << 23), b2 = b1 - (23u << 23);
  const bool ok = t >= (52 << 20);
  h = ok ? __uint_as_float(f) : 0.f;
  m = ok ? __uint_as_float(b1 | ((lo >> 6) & 0x7fffffu)) - __uint_as_float(b1) : 0.f;
  l = ok ? __uint_as_float(b2 | ((lo & 63u) << 17)) - __uint_as_float(b2) : 0.f;
}
__device__ __forceinline__ T3 t3_of(double x, double y, int bias20) {
  float xh, xm, xl, yh, ym, yl;
  t3_split(x, bias20, xh, xm, xl);
  t3_split(y, bias20, yh, ym, yl);
  return T3{f2_pack(xh, yh), f2_pack(xm, ym), f2_pack(xl, yl)};
}
// One word back to a double with the scale undone (subnormal floats are 0).
__device__ __forceinline__ double t3_word(float f, int bias20) {
  const unsigned u = __float_as_uint(f), a = u & 0x7fffffffu;
  return a >= (1u << 23) ? __hiloint2double((int)((u & 0x80000000u) | ((a >> 3) + (unsigned)bias20)), (int)(u << 29))
                         : 0.0;
}
// x half minus y half as a double with the scale undone.
__device__ __forceinline__ double t3_diff(T3 c, int bias20) {
  // the halves subtract exactly up to the last word: pack them as (x, x) - (y, y)
  float hx, hy, mx, my, lx, ly;
  f2_unpack(c.h, hx, hy);
  f2_unpack(c.m, mx, my);
  f2_unpack(c.l, lx, ly);
  float s, e, s1, e1, m, e2;
  auto two_sum = [](float a, float b, float& s_, float& e_) {
    s_ = __fadd_rn(a, b);
    const float z = __fadd_rn(s_, -a);
    e_ = __fadd_rn(__fadd_rn(a, -__fadd_rn(s_, -z)), __fadd_rn(b, -z));
  };
  two_sum(hx, -hy, s, e);
  two_sum(mx, -my, s1, e1);
  two_sum(s1, e, m, e2);
  const float l = __fadd_rn(__fadd_rn(__fadd_rn(lx, -ly), e1), e2);
  return __dadd_rn(t3_word(s, bias20), __dadd_rn(t3_word(m, bias20), t3_word(l, bias20)));
}

// (K/q0)^2 etc.: numerator and denominator of w0 Da + 2 w2 Db with the linear
// weights 0.3 : 0.6 : 0.1 of wenop divided by 0.3 (0.6f is 2 x 0.3f exactly;
// the ratio 0.1f / 0.3f to 72 bits).
__device__ __forceinline__ T3 t3_weno5_part(T3 q0, T3 q1, T3 q2, T3 Da, T3 Db) {
  const T3 ratio{f2_both(0x1.555554p-2f), f2_both(0x1.8e38e4p-27f), f2_both(0x1.2f684ap-53f)};
  const f2 K = f2_pow2_min(q0.h, q1.h, q2.h);
  const T3 a0 = t3_sqr(t3_rcp(q0, K)), a1 = t3_sqr(t3_rcp(q1, K)), a2 = t3_mul(t3_sqr(t3_rcp(q2, K)), ratio);
  const T3 S = t3_add(t3_add(a0, 2.f, a1), 1.f, a2);
  const T3 N = t3_add(t3_mul(a0, Da), 2.f, t3_mul(a2, Db));
  return t3_mul(N, t3_rcp(S, f2_both(1.f)));
}

// 6 R for both halves from the five differences d_j (WENO5); eps = 4 x the
// reference's epsilon in the scale of d^2.  The indicators are 4 x the
// reference's: 13/3 t^2 + s^2 + 4 eps, squared by t3_weno5_part.
__device__ __forceinline__ T3 t3_weno5_diff(T3 d[5], f2 eps) {
  const f2 k4 = f2_both((float)(4.0 * Lit::c13_12));  // a float exactly
#pragma unroll
  for (int j = 0; j < 5; ++j) d[j] = t3_grid(d[j]);
  auto part = [&](T3 t) { return t3_add_f(t3_mul_f(t3_sqr(t3_norm(t)), k4), eps); };
  auto square = [&](T3 a, float c, T3 b) { return t3_sqr(t3_norm(t3_lin(a, c, b))); };
  const T3 t0 = t3_lin(d[1], -1.f, d[0]), t1 = t3_lin(d[2], -1.f, d[1]);
  const T3 t2 = t3_lin(d[3], -1.f, d[2]), t3 = t3_lin(d[4], -1.f, d[3]);
  const T3 T1 = part(t1), T2 = part(t2), D1 = t3_lin(t2, -1.f, t1);
  // the difference of the two middle polynomials: d_1 - 5 d_2 - 2 d_3
  T3 R = t3_lin(t3_lin(d[1], -5.f, d[2]), -2.f, d[3]);
  {
    // (t2 - 2 d_2 = d_3 - 3 d_2, and t0 + 2 d_1 = -(d_0 - 3 d_1))
    const T3 G = t3_weno5_part(t3_add(T2, 1.f, square(d[3], -3.f, d[2])), t3_add(T1, 1.f, square(d[1], 1.f, d[2])),
                               t3_add(part(t0), 1.f, square(d[0], -3.f, d[1])), D1, t3_lin(t1, -1.f, t0));
    R = t3_add(R, -1.f, G);
  }
  const T3 G = t3_weno5_part(t3_add(part(t3), 1.f, square(d[4], -3.f, d[3])), t3_add(T2, 1.f, square(d[2], 1.f, d[3])),
                             t3_add(T1, 1.f, square(d[1], -3.f, d[2])), t3_lin(t3, -1.f, t2), D1);
  return t3_add(R, 1.f, G);
}

// 2 R of the third-order pair (rhs_hybrid_low_llf.m4:349-397): wenop on
// (b, c, d) is (c + d - w1 t) / 2 with t = b - 2c + d, linear weights 2/3 and
// 1/3 (their single-precision literals are in the ratio 2 : 1 exactly).  The
// three differences d_1..d_3 give R on (x_1, x_2, x_3) minus (x_2, x_3, x_4).
__device__ __forceinline__ T3 t3_weno3_part(T3 q0, T3 q1, T3 t) {
  const f2 K = f2_pow2_min(q0.h, q1.h);
  const T3 a0 = t3_sqr(t3_rcp(q0, K)), a1 = t3_sqr(t3_rcp(q1, K));
  return t3_mul(t3_mul(a1, t), t3_rcp(t3_add(a1, 2.f, a0), f2_both(1.f)));
}
__device__ __forceinline__ T3 t3_weno3_diff(const T3 d[3], f2 eps) {
  const T3 q1 = t3_add_f(t3_sqr(d[0]), eps), q2 = t3_add_f(t3_sqr(d[1]), eps), q3 = t3_add_f(t3_sqr(d[2]), eps);
  const T3 lo = t3_weno3_part(q2, q1, t3_add(d[1], -1.f, d[0]));
  const T3 hi = t3_weno3_part(q3, q2, t3_add(d[2], -1.f, d[1]));
  // -(d_2 + d_3) + w t (hi) - w t (lo)
  return t3_add(t3_add(hi, -1.f, lo), -1.f, t3_add(d[1], 1.f, d[2]));
}

// Flux difference of one field along one direction at one cell, without the
// factor 1/6 (order 5) or 1/2 (order 3): w points at the field and f at half
// its flux at the cell, sw and sf are the strides along the direction, ha is
// half the split speed.  Values of any magnitude; a non-finite difference
// gives NaN.  Out of line: one copy of the code for the ten calls of a cell.
template <int ORDER>
__device__ __noinline__ double weno_flux64(const double* w, int sw, const double* f, int sf, double ha) {
  constexpr int N = ORDER == 5 ? 5 : 3;   // differences per sign
  constexpr int O = ORDER == 5 ? 3 : 2;   // points before the cell
  double dx[N], dy[N];
  unsigned top = 0;
  {
    double dw[N + 1], df[N + 1];
    double w0 = w[-O * sw], f0 = f[-O * sf];
#pragma unroll
    for (int j = 0; j <= N; ++j) {
      const double w1 = w[(j + 1 - O) * sw], f1 = f[(j + 1 - O) * sf];
      dw[j] = __dsub_rn(w1, w0);
      df[j] = __dsub_rn(f1, f0);
      w0 = w1;
      f0 = f1;
    }
    // x_{j+1} - x_j, and y_{j+1} - y_j = m_{N-j} - m_{N+1-j} (mirrored)
#pragma unroll
    for (int j = 0; j < N; ++j) {
      dx[j] = fma(ha, dw[j], df[j]);
      dy[j] = fma(ha, dw[N - j], -df[N - j]);
      top = max(top, max((unsigned)__double2hiint(dx[j]) & 0x7fffffffu, (unsigned)__double2hiint(dy[j]) & 0x7fffffffu));
    }
  }
  if (top == 0u) return 0.0;  // every difference 0 (or below 2^-1042)
  if (top >= 0x7ff00000u) return __longlong_as_double(0x7ff8000000000000LL);
  const int E = max((int)(top >> 20), 128), bias20 = (E - 127) << 20;
  // epsilon (a float exactly, with the factor 4 of order 5) in the scale
  // 2^(2 (1023 - E)); at the ends of its range it is far above or below every
  // indicator, and the weights no longer depend on it
  const unsigned e0 = __float_as_uint((float)(ORDER == 5 ? 4.0 * Lit::weno_eps : Lit::weno_eps));
  const int ee = min(max((int)(e0 >> 23) - 2 * (E - 1023), 7), 227);
  const f2 eps = f2_both(__uint_as_float((e0 & 0x7fffffu) | ((unsigned)ee << 23)));
  T3 d[N];
#pragma unroll
  for (int j = 0; j < N; ++j) d[j] = t3_of(dx[j], dy[j], bias20);
  if constexpr (ORDER == 5) return t3_diff(t3_weno5_diff(d, eps), bias20);
  else return t3_diff(t3_weno3_diff(d, eps), bias20);
}

}  // namespace enl
