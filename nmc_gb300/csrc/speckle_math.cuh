// speckle_math.cuh - the functions of the speckle post-processing in pairs of
// floats (hi + lo, about 44 bits: two-sum and fused two-product, Dekker 1971 and
// Knuth).  Each is evaluated to 2^-31 of its value or better and rounded once,
// so its result is within 0.51 units in the last place, as a double function's
// rounded to float is; arguments outside the range that the pairs cover take the
// double expressions.  Host code may compile this file (with the rounding
// intrinsics defined), which is how each bound is tested.
#pragma once

namespace nmc {

struct FF {
  float h, l;
};
__device__ __forceinline__ FF two_sum(float a, float b) {
  const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
  return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t))};
}
__device__ __forceinline__ FF fast_two_sum(float a, float b) {  // |a| >= |b|
  const float s = __fadd_rn(a, b);
  return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ FF two_prod(float a, float b) {
  const float p = __fmul_rn(a, b);
  return {p, __fmaf_rn(a, b, -p)};
}

// pi as three floats: hi + mid + lo
constexpr float kPi1 = 3.14159274f, kPi2 = -8.74227766e-8f, kPi3 = -3.43e-15f;

// x - k unit pi for a small integer k (unit = 2 or 1/2): the product with the
// leading float is exact as a pair, and x lies within a factor of two of it
__device__ __forceinline__ FF reduce_pi(float x, float k, float unit) {
  const FF p = two_prod(k, unit * kPi1);
  const FF r = two_sum(__fsub_rn(x, p.h), -p.l);
  const FF q = two_prod(k, unit * kPi2);
  const FF t = two_sum(r.h, -q.h);
  return fast_two_sum(t.h, t.l + (r.l - q.l) - k * (unit * kPi3));
}

__device__ __noinline__ float wrap_slow(float a) { return (float)atan2(sin((double)a), cos((double)a)); }

// atan2(sin a, cos a): a - 2 pi k in (-pi, pi]
__device__ __forceinline__ float wrap_ref(float a) {
  const float m = fabsf(a);
  if (m < kPi1) return a;             // the floats below kPi1 are below pi
  if (!(m < 4096.f)) return wrap_slow(a);
  FF r = reduce_pi(a, rintf(a * (0.5f / kPi1)), 2.f);
  const float s = copysignf(1.f, r.h);
  if (fabsf(r.h) > kPi1 || (fabsf(r.h) == kPi1 && s * r.l > kPi2)) {  // beyond +-pi: one turn back
    const FF t = two_sum(r.h, -s * (2.f * kPi1));
    r = fast_two_sum(t.h, t.l + (r.l - s * (2.f * kPi2)));
  }
  return r.h;
}

// a (bh + bl) for pairs of floats
__device__ __forceinline__ FF mul(FF a, FF b) {
  const FF p = two_prod(a.h, b.h);
  return {p.h, p.l + fmaf(a.h, b.l, a.l * b.h)};
}
// c (as a pair) + t, |c| >= |t|
__device__ __forceinline__ FF lead(float ch, float cl, float t) {
  const FF s = fast_two_sum(ch, t);
  return {s.h, s.l + cl};
}
// 1/6 and 1/24 as two floats
constexpr float kSixth1 = 0.166666672f, kSixth2 = -4.96705388e-9f, k24th1 = 0.0416666679f, k24th2 = -1.24176347e-9f;

// sin x for |x| <= 4, by reduction to [-pi/4, pi/4] and the Taylor series.  Its
// first three terms are pairs, the rest, at most 1/30 of the third, floats: the
// value is good to 2^-31 before its one rounding.
__device__ __forceinline__ float sin_ref(float x) {
  const float k = rintf(x * (2.f / kPi1));
  const FF y = k == 0.f ? FF{x, 0.f} : reduce_pi(x, k, 0.5f);
  const FF z = mul(y, y);
  const int q = (int)k & 3;
  float v;
  if (q & 1) {  // cos y = 1 - z/2 + z^2 (1/24 - z/720 + ...)
    const float c = fmaf(fmaf(fmaf(2.08767559e-9f, z.h, -2.75573192e-7f), z.h, 2.48015873e-5f), z.h, -1.38888889e-3f);
    const FF w = mul(mul(z, z), lead(k24th1, k24th2, c * z.h));
    const FF a = fast_two_sum(1.f, -0.5f * z.h), b = two_sum(a.h, w.h);
    v = b.h + (b.l + (a.l + fmaf(-0.5f, z.l, w.l)));
  } else {  // sin y = y - y z (1/6 - z/120 + ...)
    const float c = fmaf(fmaf(fmaf(2.50521079e-8f, z.h, -2.75573192e-6f), z.h, 1.98412698e-4f), z.h, -8.33333333e-3f);
    const FF w = mul(mul(y, z), lead(kSixth1, kSixth2, c * z.h));
    const FF a = fast_two_sum(y.h, -w.h);
    v = a.h + (a.l + (y.l - w.l));
  }
  return q & 2 ? -v : v;
}

// e^a for a <= 0: 2^n e^r with r in [-ln 2 / 2, ln 2 / 2] and the Taylor series,
// its first four terms as pairs
__device__ __forceinline__ float exp_ref(float a) {
  if (!(a > -87.f)) return (float)exp((double)a);  // NaN, or below the normal floats
  constexpr float kLn1 = 0.693147182f, kLn2 = -1.90465421e-9f;  // ln 2 as two floats
  const float n = rintf(a * 1.44269504f);
  const FF p = two_prod(n, kLn1);
  const FF r = two_sum(__fsub_rn(a, p.h), -fmaf(n, kLn2, p.l));
  const float c = fmaf(fmaf(fmaf(fmaf(fmaf(2.75573192e-6f, r.h, 2.48015873e-5f), r.h, 1.98412698e-4f), r.h, 1.38888889e-3f), r.h,
                            8.33333333e-3f), r.h, 4.16666667e-2f);
  const FF s = mul(r, r);
  const FF w = mul(mul(s, r), lead(kSixth1, kSixth2, c * r.h));
  const FF t = fast_two_sum(1.f, r.h), u = two_sum(t.h, 0.5f * s.h), v = two_sum(u.h, w.h);
  return (v.h + (v.l + (u.l + (t.l + (r.l + fmaf(0.5f, s.l, w.l)))))) * __int_as_float((127 + (int)n) << 23);
}

__device__ __noinline__ float interfere_slow(float a, float c, float interf, float env) {
  const double two = 2.0;  // MC_TWO (definitions.h:60)
  return (float)(((double)(a + c) + two * sqrt((double)(a * c)) * interf * env) / 4.0f);
}

// (a + c + 2 sqrt(a c) interf env) / 4; a product whose square root has no
// normal float as its remainder (p below 2^-100) goes the slow way
__device__ __forceinline__ float interfere(float a, float c, float interf, float env) {
  const float p = a * c;
  if (!((p == 0.f || p > 1e-30f) && fabsf(a) < 1e15f && fabsf(c) < 1e15f)) return interfere_slow(a, c, interf, env);
  const float s = __fsqrt_rn(p);
  const float sl = s > 0.f ? __fdividef(__fmaf_rn(-s, s, p), 2.f * s) : 0.f;
  const FF w = two_prod(interf, env);
  const FF u = two_prod(s, w.h);
  const FF t = two_sum(a + c, 2.f * u.h);
  return 0.25f * (t.h + (t.l + 2.f * (u.l + fmaf(s, w.l, sl * w.h))));
}

}  // namespace nmc
