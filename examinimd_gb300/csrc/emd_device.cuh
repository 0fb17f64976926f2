// Device-side helpers shared by the kernel files.
#pragma once
#include <cuda_runtime.h>

namespace emd {

constexpr unsigned FULL_MASK = 0xffffffffu;

__device__ __forceinline__ void latch_status(unsigned* status, unsigned bits) {
  if (status) atomicOr(status, bits);
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(FULL_MASK, v, o);
  return v;
}

__device__ __forceinline__ int warp_sum_int(int v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(FULL_MASK, v, o);
  return v;
}

// Block-wide sum in a fixed order (lane tree, then warp tree); result valid
// in thread 0.  `sh` needs blockDim.x/32 doubles.
__device__ __forceinline__ double block_sum(double v, double* sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  v = warp_sum(v);
  if (lane == 0) sh[w] = v;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  double t = 0.0;
  if (w == 0) {
    t = lane < nw ? sh[lane] : 0.0;
    t = warp_sum(t);
  }
  __syncthreads();
  return t;
}

// ------------------------------------------------- FP32 view of a double
// Truncation to FP32 by integer operations: magnitudes below 2^-126 become 0,
// beyond the FP32 range (and NaN) infinity.  Within 2^-23 relative otherwise.
__device__ __forceinline__ float f32_bits(double v) {
  const unsigned hi = __double2hiint(v), lo = __double2loint(v);
  const unsigned e = (hi >> 20) & 0x7ffu;
  unsigned m = (((hi & 0x7fffffffu) << 3) | (lo >> 29)) - 0xc0000000u;  // exponent less 896
  m = e < 897u ? 0u : (e > 1150u ? 0x7f800000u : m);
  return __uint_as_float(m | (hi & 0x80000000u));
}
__device__ __forceinline__ double f64_of_normal(float f) {  // exact for a normal f > 0
  const unsigned b = __float_as_uint(f);
  return __hiloint2double(int((b >> 3) + 0x38000000u), int(b << 29));
}

// IEEE 1 / d.  For d within [2^-96, 2^96] whose significand is not all ones: an
// FP32 reciprocal (2^-21 off), one cubic step in FP64 and Markstein's final
// correction y + y (1 - d y), which returns the correctly rounded reciprocal
// for every other significand (P. Markstein, IBM J. Res. Dev. 34 (1990) 111):
// five FP64 instructions.  Everything else takes the divide, out of line.
static __device__ __noinline__ double recip_div(double d) { return 1.0 / d; }
__device__ __forceinline__ double recip_rn(double d) {
  const unsigned hi = __double2hiint(d);
  const bool plain = hi - 0x39f00000u < 0x0c000000u &&
                     !((hi & 0xfffffu) == 0xfffffu && unsigned(__double2loint(d)) == 0xffffffffu);
  if (!plain) return recip_div(d);
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(f32_bits(d)));
  const double r0 = f64_of_normal(r);
  const double e = __fma_rn(-d, r0, 1.0);
  const double y = __fma_rn(r0, __fma_rn(e, e, e), r0);
  return __fma_rn(y, __fma_rn(-d, y, 1.0), y);
}

// Threshold for an FP32 r^2 formed from f32_bits positions: every partner with
// r^2 < cutsq lies below it.  Such a partner has coordinates below M in
// magnitude, so the FP32 differences are off by at most d = 2^-21 M per
// dimension and r^2 by 2 sqrt(3) rc d + 3 d^2 plus the FP32 operations'
// rounding.  Non-finite coordinates give a comparison that rejects nothing.
__device__ __forceinline__ float f32_cut_threshold(float cutsq, float x, float y, float z) {
  const float rc = sqrtf(cutsq);
  const float d = (fmaxf(fabsf(x), fmaxf(fabsf(y), fabsf(z))) + rc) * 4.7683716e-7f;
  return fmaf(cutsq, 1.00001f, fmaf(4.0f * rc, d, 3.0f * d * d));
}

}  // namespace emd
