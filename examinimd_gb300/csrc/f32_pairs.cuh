// Sums of products in FP32 pairs (high and low part, 48 bits) on the FP32 pipe,
// which issues 76 times as many lane operations as the FP64 one here.
#pragma once

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

// 1.5 times a power of two at least four times as large as b: sums below 2 b in
// magnitude leave it within one binade
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
