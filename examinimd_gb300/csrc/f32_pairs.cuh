// Sums of products in FP32 pairs (high and low part, 48 bits) on the FP32 pipe,
// which issues 76 times as many lane operations as the FP64 one here.  Built from
// Knuth's two-sum and Dekker's product (here a fused multiply-add's remainder).
#pragma once
#include "emd_device.cuh"

namespace emd {

struct F2 {
  float h, l;
};

// plain roundings, whatever the compiler may fuse
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }

// h + l renormalised, |h| >= |l| or h = 0
__device__ __forceinline__ F2 f2_norm(float h, float l) {
  const float s = add_rn(h, l);
  return F2{s, sub_rn(l, sub_rn(s, h))};
}

// a + b and what its rounding leaves off (Knuth's two-sum)
__device__ __forceinline__ F2 f2_two_sum(float a, float b) {
  const float t = add_rn(a, b), y = sub_rn(t, a);
  return F2{t, add_rn(sub_rn(a, sub_rn(t, y)), sub_rn(b, y))};
}

// 1.5 times the power of two that is four times b's own (more than twice b): sums up
// to b in magnitude leave it within one binade
__device__ __forceinline__ float f2_base(float b) {
  const unsigned e = min(max((__float_as_uint(b) >> 23) & 0xffu, 67u), 250u) + 2u;
  return __uint_as_float((e << 23) | 0x400000u);
}

// Sum of products on the grid of a base: s = base + the products rounded to the
// base's last place one after another, c = what that left out, which is exact
// (the difference of two neighbouring s and the product less it), plus the
// cross terms.  Six operations a product.
struct F2Sum {
  float s, c;
  __device__ __forceinline__ void add(F2 a, F2 b) {
    const float t = fmaf(a.h, b.h, s);
    const float r = fmaf(a.h, b.h, -sub_rn(t, s));
    c = fmaf(a.h, b.l, c);
    c = fmaf(a.l, b.h, c);
    c = add_rn(c, r);
    s = t;
  }
  __device__ __forceinline__ F2 value(float base) const { return f2_norm(sub_rn(s, base), c); }
};

// p + i r times a + i b (nb = -b); base: f2_base of the factors' product
__device__ __forceinline__ void f2_cmul(F2& p, F2& r, F2 a, F2 b, F2 nb, float base) {
  F2Sum pn{base, 0.f}, rn{base, 0.f};
  pn.add(p, a);
  pn.add(r, nb);
  rn.add(p, b);
  rn.add(r, a);
  p = pn.value(base);
  r = rn.value(base);
}

// A double as a pair, by integer operations (conversions run at the FP64 rate
// here): truncated to 24 bits and the 29 bits below, within 2^-47; magnitudes
// below 2^-75 have no low part, below 2^-126 are 0, beyond the FP32 range infinite.
__device__ __forceinline__ F2 f2_split(double v) {
  const unsigned hi = __double2hiint(v), lo = __double2loint(v);
  const int e = int(hi >> 20 & 0x7ffu) - 948;  // exponent of the last of the 52 bits, biased
  const float s = e > 0 && e < 255 ? __uint_as_float(unsigned(e) << 23 | (hi & 0x80000000u)) : 0.f;
  return F2{f32_bits(v), __uint2float_rn(lo & 0x1fffffffu) * s};
}

__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
  const float h = __fmul_rn(a.h, b.h);
  return F2{h, fmaf(a.l, b.h, fmaf(a.h, b.l, fmaf(a.h, b.h, -h)))};
}
// a + b; c + a with |c.h| >= |a.h|
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
  const float t = add_rn(a.h, b.h), y = sub_rn(t, a.h);
  const float d = add_rn(sub_rn(a.h, sub_rn(t, y)), sub_rn(b.h, y));
  return f2_norm(t, add_rn(d, add_rn(a.l, b.l)));
}
__device__ __forceinline__ F2 f2_onto(F2 c, F2 a) {
  const float t = add_rn(c.h, a.h);
  return F2{t, add_rn(sub_rn(a.h, sub_rn(t, c.h)), add_rn(c.l, a.l))};
}

// 1 / sqrt(a): a step of Newton's iteration, to second order, from the FP32 value
__device__ __forceinline__ F2 f2_rsqrt(F2 a) {
  const float y = rsqrtf(a.h);
  const F2 t = f2_mul(a, f2_mul(F2{y, 0.f}, F2{y, 0.f}));
  const float e = sub_rn(sub_rn(1.f, t.h), t.l);
  return f2_norm(y, y * fmaf(0.375f * e, e, 0.5f * e));
}

// sin(x) and cos(x) for |x| up to a few hundred: x less a multiple of pi / 2 (three
// FP32 parts), then the Taylor series to x^15 and x^14, the terms that reach below
// 2^-24 of the result in FP32.  Within 2^-44.
__device__ __forceinline__ void f2_sincos(F2 x, F2& sn, F2& cs) {
  constexpr double kHalfPi = 1.57079632679489661923;
  constexpr float p1 = float(kHalfPi), p2 = float(kHalfPi - double(p1)), p3 = float(kHalfPi - double(p1) - double(p2));
  const float k = rintf(x.h * float(1.0 / kHalfPi));
  const float h1 = __fmul_rn(k, p1), e1 = fmaf(k, p1, -h1), h2 = __fmul_rn(k, p2), e2 = fmaf(k, p2, -h2);
  const F2 r = f2_add(f2_add(f2_norm(x.h, x.l), F2{-h1, -e1}), F2{-h2, -fmaf(k, p3, e2)});
  const F2 z = f2_mul(r, r);
  auto c = [](double v) { return F2{float(v), float(v - double(float(v)))}; };
  const float ts = fmaf(z.h, fmaf(z.h, fmaf(z.h, float(-1.0 / 1307674368000.0), float(1.0 / 6227020800.0)),
                                  float(-1.0 / 39916800.0)), float(1.0 / 362880.0));
  const float tc = fmaf(z.h, fmaf(z.h, float(-1.0 / 87178291200.0), float(1.0 / 479001600.0)), float(-1.0 / 3628800.0));
  F2 s = f2_onto(c(-1.0 / 5040.0), F2{z.h * ts, 0.f});
  s = f2_onto(c(1.0 / 120.0), f2_mul(z, s));
  s = f2_onto(c(-1.0 / 6.0), f2_mul(z, s));
  s = f2_onto(r, f2_mul(f2_mul(r, z), s));
  F2 o = f2_onto(c(1.0 / 40320.0), F2{z.h * tc, 0.f});
  o = f2_onto(c(-1.0 / 720.0), f2_mul(z, o));
  o = f2_onto(c(1.0 / 24.0), f2_mul(z, o));
  o = f2_onto(c(-0.5), f2_mul(z, o));
  o = f2_onto(c(1.0), f2_mul(z, o));
  s = f2_norm(s.h, s.l);
  o = f2_norm(o.h, o.l);
  const int n = int(k);
  const F2 a = n & 1 ? o : s, b = n & 1 ? s : o;  // sin, cos but for the signs
  const float ga = n & 2 ? -1.f : 1.f, gb = (n + 1) & 2 ? -1.f : 1.f;
  sn = F2{ga * a.h, ga * a.l};
  cs = F2{gb * b.h, gb * b.l};
}

// s + c += a b
__device__ __forceinline__ void f2_dot(F2& s, F2 a, F2 b) {
  const float h = __fmul_rn(a.h, b.h), e = fmaf(a.h, b.h, -h);
  const float t = add_rn(s.h, h), y = sub_rn(t, s.h);
  const float d = add_rn(sub_rn(s.h, sub_rn(t, y)), sub_rn(h, y));
  s.l = fmaf(a.h, b.l, s.l);
  s.l = fmaf(a.l, b.h, s.l);
  s.l = add_rn(s.l, add_rn(d, e));
  s.h = t;
}
// a + b + c, rounded
__device__ __forceinline__ float f2_sum(F2 a, F2 b, float c) {
  const float t = add_rn(a.h, b.h), y = sub_rn(t, a.h);
  const float d = add_rn(sub_rn(a.h, sub_rn(t, y)), sub_rn(b.h, y));
  const float z = add_rn(t, c), x = sub_rn(z, t);
  const float f = add_rn(sub_rn(t, sub_rn(z, x)), sub_rn(c, x));
  return add_rn(z, add_rn(add_rn(f, d), add_rn(a.l, b.l)));
}

}  // namespace emd
