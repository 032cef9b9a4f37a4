// Double-float ("df") arithmetic: a value is hi + lo with two FP32 numbers,
// |lo| <= ulp(hi) / 2, about 48 significant bits.  GB300 runs FP32 at 64x its
// FP64 rate, so FP64-class quadrature is cheaper in df on the FP32 pipes.
//
// Building blocks (published methods):
//   * TwoSum (Knuth), Fast2Sum (Dekker), TwoProduct via FMA - error-free
//     transformations;
//   * the "sloppy" df addition of Dekker / Bailey's double-double libraries
//     (error ~2^-47 of |a| + |b|) and the FMA-based df product;
//   * square root and reciprocal from the FP32 approximation: one Newton step
//     in FP32 to a value accurate to its last bit, one more for the low part
//     (Karp-Markstein form);
//   * sums of products in unnormalized accumulators (the compensated dot
//     product of Ogita, Rump and Oishi): 12 FP32 operations a term against 18
//     of a df product and a df addition, the same rounding behaviour over the
//     ~100 terms of a quadrature rule;
//   * polynomials by a Horner step that knows |c| >= |p s|: 9 operations
//     against 18;
//   * sin, cos on [-pi/4, pi/4] and exp on [-ln2/2, ln2/2] by their Taylor
//     series (argument reduction by Cody-Waite in FP64 by the caller), the
//     high-order terms in FP32 where they are below 2^-25 of the result.
#pragma once

#include <cuda_runtime.h>

#include "df_constants.h"

namespace {

struct df {
  float hi, lo;
};

__device__ __forceinline__ df df_make(double x) {
  const float h = (float)x;
  return {h, (float)(x - (double)h)};
}
__device__ __forceinline__ double df_to_double(df a) { return (double)a.hi + (double)a.lo; }

__device__ __forceinline__ df two_sum(float a, float b) {
  const float s = a + b;
  const float bb = s - a;
  return {s, (a - (s - bb)) + (b - bb)};
}
__device__ __forceinline__ df fast_two_sum(float a, float b) {  // |a| >= |b| or a == 0
  const float s = a + b;
  return {s, b - (s - a)};
}

__device__ __forceinline__ df df_add(df a, df b) {
  df s = two_sum(a.hi, b.hi);
  s.lo += a.lo + b.lo;
  return fast_two_sum(s.hi, s.lo);
}
__device__ __forceinline__ df df_neg(df a) { return {-a.hi, -a.lo}; }
__device__ __forceinline__ df df_sub(df a, df b) { return df_add(a, df_neg(b)); }
__device__ __forceinline__ df df_add_f(df a, float b) {
  df s = two_sum(a.hi, b);
  s.lo += a.lo;
  return fast_two_sum(s.hi, s.lo);
}
__device__ __forceinline__ df df_mul(df a, df b) {
  const float p = a.hi * b.hi;
  float e = fmaf(a.hi, b.hi, -p);
  e = fmaf(a.hi, b.lo, e);
  e = fmaf(a.lo, b.hi, e);
  return fast_two_sum(p, e);
}
__device__ __forceinline__ df df_sqr(df a) {
  const float p = a.hi * a.hi;
  float e = fmaf(a.hi, a.hi, -p);
  e = fmaf(2.f * a.hi, a.lo, e);
  return fast_two_sum(p, e);
}
// a * 2^k for a float power of two p2 (exact)
__device__ __forceinline__ df df_scale2(df a, float p2) { return {a.hi * p2, a.lo * p2}; }

// sqrt(a), a > 0: s = a.hi * r (r ~ 1/sqrt(a.hi)) refined to FP32 accuracy,
// then the low part from a - s^2.
__device__ __forceinline__ df df_sqrt(df a) {
  const float r = rsqrtf(a.hi), h = 0.5f * r;
  const float s = a.hi * r;
  const float s1 = fmaf(h, fmaf(-s, s, a.hi), s);
  const float e = fmaf(-s1, s1, a.hi) + a.lo;
  return fast_two_sum(s1, h * e);
}
// 1 / a: r = 1/a.hi, then r + r (1 - a r).
__device__ __forceinline__ df df_rcp(df a) {
  const float r = __frcp_rn(a.hi);
  const float e = fmaf(-a.lo, r, fmaf(-a.hi, r, 1.f));
  return fast_two_sum(r, r * e);
}
// R = sqrt(a) and 1/R at once, from one FP32 reciprocal square root.
__device__ __forceinline__ void df_sqrt_rcp(df a, df &R, df &Ri) {
  const float r = rsqrtf(a.hi), h = 0.5f * r;
  const float s = a.hi * r;
  const float s1 = fmaf(h, fmaf(-s, s, a.hi), s);
  const float e = fmaf(-s1, s1, a.hi) + a.lo;
  R = fast_two_sum(s1, h * e);
  const float r1 = fmaf(r, fmaf(-R.hi, r, 1.f), r);
  const float d = fmaf(-R.lo, r1, fmaf(-R.hi, r1, 1.f));
  Ri = fast_two_sum(r1, r1 * d);
}

// a - b without the final normalization: the low part may exceed half an ulp
// of a high part that cancelled, which products of the difference tolerate.
__device__ __forceinline__ df df_diff(df a, df b) {
  const float s = a.hi - b.hi, t = s - a.hi;
  return {s, ((a.hi - (s - t)) - (b.hi + t)) + (a.lo - b.lo)};
}
// x^2 + y^2 + z^2 of unnormalized differences.
__device__ __forceinline__ df df_sumsq(df x, df y, df z) {
  const float px = x.hi * x.hi, py = y.hi * y.hi, pz = z.hi * z.hi;
  const float ex = fmaf(x.hi + x.hi, x.lo, fmaf(x.hi, x.hi, -px));
  const float ey = fmaf(y.hi + y.hi, y.lo, fmaf(y.hi, y.hi, -py));
  const float ez = fmaf(z.hi + z.hi, z.lo, fmaf(z.hi, z.hi, -pz));
  const df s = two_sum(px, py), t = two_sum(s.hi, pz);
  return fast_two_sum(t.hi, (s.lo + t.lo) + (ex + (ey + ez)));
}
// acc += x y, acc unnormalized (df_fin normalizes it).
__device__ __forceinline__ void df_mac(df &acc, df x, df y) {
  const float p = x.hi * y.hi;
  float e = fmaf(x.hi, y.hi, -p);
  e = fmaf(x.hi, y.lo, e);
  e = fmaf(x.lo, y.hi, e);
  const df s = two_sum(acc.hi, p);
  acc.hi = s.hi;
  acc.lo += s.lo + e;
}
__device__ __forceinline__ df df_fin(df a) { return fast_two_sum(a.hi, a.lo); }
// c + p s, |c.hi| >= |p s|: a Horner step; the result is unnormalized (its low
// part within about an ulp of the high one).
__device__ __forceinline__ df df_horner(df p, df s, df c) {
  const float m = p.hi * s.hi;
  float e = fmaf(p.hi, s.hi, -m);
  e = fmaf(p.hi, s.lo, e);
  e = fmaf(p.lo, s.hi, e);
  const float h = c.hi + m;
  return {h, (m - (h - c.hi)) + (e + c.lo)};
}
// The same with an FP32 p (the first step after an FP32 tail).
__device__ __forceinline__ df df_horner_f(float p, df s, df c) {
  const float m = p * s.hi;
  const float e = fmaf(p, s.lo, fmaf(p, s.hi, -m));
  const float h = c.hi + m;
  return {h, (m - (h - c.hi)) + (e + c.lo)};
}
// a b + c d.
__device__ __forceinline__ df df_dot2(df a, df b, df c, df d) {
  const float p = a.hi * b.hi, q = c.hi * d.hi;
  const float e = fmaf(a.lo, b.hi, fmaf(a.hi, b.lo, fmaf(a.hi, b.hi, -p)));
  const float f = fmaf(c.lo, d.hi, fmaf(c.hi, d.lo, fmaf(c.hi, d.hi, -q)));
  const df s = two_sum(p, q);
  return fast_two_sum(s.hi, s.lo + (e + f));
}
// a b + c.
__device__ __forceinline__ df df_muladd(df a, df b, df c) {
  const float p = a.hi * b.hi;
  const float e = fmaf(a.lo, b.hi, fmaf(a.hi, b.lo, fmaf(a.hi, b.hi, -p)));
  const df s = two_sum(p, c.hi);
  return fast_two_sum(s.hi, s.lo + (e + c.lo));
}

// Taylor coefficient 1/n! as df (exact values from df_constants.h).
__device__ __forceinline__ df inv_fact(int n) { return {DF_FACT_HI[n], DF_FACT_LO[n]}; }

// sin r, cos r for |r| <= pi/4 + a little (df): Taylor series in s = r^2,
// sin up to r^17, cos up to r^18; terms below 2^-25 of the result in FP32.
// sm: sin r - r, accurate relative to itself.
__device__ __forceinline__ void df_sincos_reduced(df r, df &sn, df &cs, df &sm) {
  const df s = df_sqr(r);
  const float sf = s.hi;
  // FP32 tails: sin coefficients of r^17 .. r^11, cos of r^18 .. r^12 (signs alternate)
  float ts = -inv_fact(17).hi;
  ts = fmaf(ts, sf, inv_fact(15).hi);
  ts = fmaf(ts, sf, -inv_fact(13).hi);
  ts = fmaf(ts, sf, inv_fact(11).hi);
  float tc = inv_fact(18).hi;
  tc = fmaf(tc, sf, -inv_fact(16).hi);
  tc = fmaf(tc, sf, inv_fact(14).hi);
  tc = fmaf(tc, sf, -inv_fact(12).hi);
  // df Horner for the leading terms
  df ps = df_horner_f(ts, s, df_neg(inv_fact(9)));
  ps = df_horner(ps, s, inv_fact(7));
  ps = df_horner(ps, s, df_neg(inv_fact(5)));
  ps = df_horner(ps, s, inv_fact(3));
  // ps = 1/3! - s/5! + ...: sin = r - r s ps
  sm = df_mul(df_neg(ps), df_mul(r, s));
  sn = {r.hi + sm.hi, 0.f};
  sn = fast_two_sum(sn.hi, (sm.hi - (sn.hi - r.hi)) + (r.lo + sm.lo));
  df pc = df_horner_f(tc, s, inv_fact(10));
  pc = df_horner(pc, s, df_neg(inv_fact(8)));
  pc = df_horner(pc, s, inv_fact(6));
  pc = df_horner(pc, s, df_neg(inv_fact(4)));
  pc = df_horner(pc, s, inv_fact(2));
  // cos = 1 - s (1/2! - s/4! + ...)
  cs = df_fin(df_horner(df_neg(pc), s, {1.f, 0.f}));
}

// e^r - 1 for |r| <= 0.35 (df): Taylor series up to r^13, tail in FP32.
__device__ __forceinline__ df df_expm1_reduced(df r) {
  const float rf = r.hi;
  float t = inv_fact(13).hi;
  t = fmaf(t, rf, inv_fact(12).hi);
  t = fmaf(t, rf, inv_fact(11).hi);
  t = fmaf(t, rf, inv_fact(10).hi);
  t = fmaf(t, rf, inv_fact(9).hi);
  t = fmaf(t, rf, inv_fact(8).hi);
  df p = df_horner_f(t, r, inv_fact(7));
  p = df_horner(p, r, inv_fact(6));
  p = df_horner(p, r, inv_fact(5));
  p = df_horner(p, r, inv_fact(4));
  p = df_horner(p, r, inv_fact(3));
  p = df_horner(p, r, inv_fact(2));
  p = df_horner(p, r, {1.f, 0.f});
  return df_mul(p, r);  // r (1 + r/2 + r^2/6 + ...)
}

// (cos x, sin x) for x given in FP64 (|x| < 2^20): quadrant reduction in FP64,
// the series in df.
__device__ __forceinline__ void df_sincos(double x, df &sn, df &cs) {
  const double n = rint(x * DF_TWO_OVER_PI);
  const double r = fma(-n, DF_PIO2_LO, fma(-n, DF_PIO2_HI, x));
  df s, c, m;
  df_sincos_reduced(df_make(r), s, c, m);
  const int q = ((int)n) & 3;
  if (q == 0) { sn = s; cs = c; }
  else if (q == 1) { sn = c; cs = df_neg(s); }
  else if (q == 2) { sn = df_neg(s); cs = df_neg(c); }
  else { sn = df_neg(c); cs = s; }
}

// x - n (c0 + c1 + c2) for an integer n, |n| < 2^8, with FP32 parts of 16
// bits (exact products).  What the three leave of the constants, 6.1e-17 (pi/2) and
// 8.8e-17 (ln 2), times n is below 1/20 of x's own rounding, 2^-48 |x|.  The
// first difference is exact: x.hi and n c0 are multiples of 2^-24 for the
// smallest reduced x and their difference stays below one.
__device__ __forceinline__ df df_reduce(df x, float n, float c0, float c1, float c2) {
  const df r = two_sum(fmaf(-n, c0, x.hi), -n * c1);
  return fast_two_sum(r.hi, r.lo + fmaf(-n, c2, x.lo));
}

// (sin x, cos x) for a df argument, |x| < 200 (quadrant count below 2^8),
// everything on the FP32 pipes; sm: sin x - x, accurate relative to itself
// where x needs no reduction.
__device__ __forceinline__ void df_sincos_df(df x, df &sn, df &cs, df &sm) {
  const float n = rintf(x.hi * DF_TWO_OVER_PI_F);
  const df r = df_reduce(x, n, DF_PIO2_F0, DF_PIO2_F1, DF_PIO2_F2);
  df s, c, m;
  df_sincos_reduced(r, s, c, m);
  const int q = ((int)n) & 3;
  if (q == 0) { sn = s; cs = c; }
  else if (q == 1) { sn = c; cs = df_neg(s); }
  else if (q == 2) { sn = df_neg(s); cs = df_neg(c); }
  else { sn = df_neg(c); cs = s; }
  const df d = df_sub(sn, x);
  sm = n == 0.f ? m : d;
}
__device__ __forceinline__ void df_sincos_df(df x, df &sn, df &cs) {
  df sm;
  df_sincos_df(x, sn, cs, sm);
}

// e^x for a df argument, -85 < x < 85, on the FP32 pipes; m1: e^x - 1,
// accurate relative to itself where x needs no reduction.
__device__ __forceinline__ df df_exp_df(df x, df &m1) {
  const float n = rintf(x.hi * DF_LOG2E_F);
  const df r = df_reduce(x, n, DF_LN2_F0, DF_LN2_F1, DF_LN2_F2);
  const df em1 = df_expm1_reduced(r);
  const df e = df_scale2(df_add_f(em1, 1.f), __int_as_float((127 + (int)n) << 23));
  const df d = df_add_f(e, -1.f);
  m1 = n == 0.f ? em1 : d;
  return e;
}
__device__ __forceinline__ df df_exp_df(df x) {
  df m1;
  return df_exp_df(x, m1);
}

__device__ __forceinline__ df df_abs(df a) { return a.hi < 0.f ? df_neg(a) : a; }

// log x, x > 0 with e^-85 < x < e^85: y0 = logf(x) (FP32), then one Newton
// step on e^y = x: t = x e^-y0 - 1 (small), log x = y0 + log(1 + t) with
// log(1 + t) = t - t^2/2 (the t^3 term is below 2^-48 for |t| < 2^-20).
__device__ __forceinline__ df df_log(df x) {
  const float y0 = logf(x.hi);
  const df e = df_exp_df({-y0, 0.f});
  const df t = df_add_f(df_mul(x, e), -1.f);
  const df u = df_add_f(t, -0.5f * t.hi * t.hi);
  return df_add_f(u, y0);
}

// atan2(y, x), (x, y) != (0, 0): t0 = atan2f(y, x) (FP32), then the exact
// correction t = t0 + atan(r), r = (y cos t0 - x sin t0) / (x cos t0 + y sin t0),
// with atan(r) = r for |r| < 2^-20 (the r^3 / 3 term is below 2^-60).
__device__ __forceinline__ df df_atan2(df y, df x) {
  const float t0 = atan2f(y.hi, x.hi);
  df s, c;
  df_sincos_df({t0, 0.f}, s, c);
  const df num = df_sub(df_mul(y, c), df_mul(x, s));
  const df den = df_add(df_mul(x, c), df_mul(y, s));
  if (den.hi == 0.f) return {t0, 0.f};
  return df_add_f(df_mul(num, df_rcp(den)), t0);
}

}  // namespace
