// FP32 sine, cosine and angle of the stage-2 kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "atan_poly.h"
#include "sincos_poly.h"

namespace ps2 {

// sin and cos of an FP32 phase (the phase ramps of binning and of the row
// refinements): Cody and Waite's reduction by pi/2 ("Software Manual for the
// Elementary Functions", 1980) with pi/2 split in three FP32 parts, each
// removed by one FMA, then minimax polynomials on [-pi/4, pi/4]
// (sincos_poly.h, fitted by make_sincos_poly.py) and the quadrant's swap and
// signs. Largest absolute error 9.2e-8 for |x| <= 5000, the FP32 rounding of a
// unit phasor; about 20 instructions. sin(+-0) = +-0; NaN and inf give NaN.
__device__ __forceinline__ void sincos_cw(float x, float* s, float* c) {
  const float k = rintf(x * kTwoOverPi);
  float r = fmaf(-k, kHalfPi1, x);
  r = fmaf(-k, kHalfPi2, r);
  r = fmaf(-k, kHalfPi3, r);
  const float u = r * r;
  float sv = fmaf(r * u, fmaf(fmaf(kSinS3, u, kSinS2), u, kSinS1), r);
  const float cv = fmaf(u * u, fmaf(fmaf(kCosQ3, u, kCosQ2), u, kCosQ1), fmaf(-0.5f, u, 1.f));
  if (x == 0.f) sv = x;
  const int q = __float2int_rn(k);
  const float s1 = (q & 1) ? cv : sv, c1 = (q & 1) ? sv : cv;
  *s = (q & 2) ? -s1 : s1;
  *c = ((q + 1) & 2) ? -c1 : c1;
}
// atan2(y, x) in FP32 for the topofit refinement's residual angles: t =
// min(|x|, |y|) / max(|x|, |y|) in [0, 1], atan t by a minimax polynomial in
// t^2 (atan_poly.h, fitted by make_atan_poly.py, 4.9e-8), then the octant's
// reflections and the sign of y. Largest absolute error 3.1e-7 (near +-pi,
// where an FP32 ulp is 2.4e-7); atan2(+-0, +0) = +-0, atan2(+-0, x < 0) = +-pi.
__device__ __forceinline__ float atan2_poly(float y, float x) {
  const float ax = fabsf(x), ay = fabsf(y);
  const float mn = fminf(ax, ay), mx = fmaxf(ax, ay);
  const float t = mx > 0.f ? __fdiv_rn(mn, mx) : 0.f;
  const float u = t * t;
  float p = fmaf(kAtanA7, u, kAtanA6);
  p = fmaf(p, u, kAtanA5);
  p = fmaf(p, u, kAtanA4);
  p = fmaf(p, u, kAtanA3);
  p = fmaf(p, u, kAtanA2);
  p = fmaf(p, u, kAtanA1);
  float r = fmaf(t * u, p, t);
  if (ay > ax) r = kHalfPiF - r;
  if (x < 0.f) r = kPiF - r;
  return copysignf(r, y);
}
__device__ __forceinline__ float2 both(const float v) { return make_float2(v, v); }

// Square roots by one step of Heron's iteration in the form Markstein gives it for
// machines with a fused multiply-add ("Computation of elementary functions on the IBM
// RISC System/6000 processor", IBM J. Res. Dev. 34, 1990): with y ~ 1 / sqrt(q) and
// s = q y, s + (q - s^2) / (2 s) is taken as s + (q - s^2) (y / 2). An approximation
// good to 2^-22 leaves an error of its square before the last rounding. The residual
// is exact in one FMA: its last bit is no lower than that of s^2, 2^-146 for q >=
// 2^-100, and FP32 goes to 2^-149. Equal to sqrtf for every float in [2^-100,
// infinity) (tests/test_gpu_sqrt.py compares them all); other values take sqrtf itself.
// sqrtf in its place made magnitudes a fifth of a window's time.
constexpr uint32_t kSqrtLo = 0x0d800000u;                // 2^-100
constexpr uint32_t kSqrtSpan = 0x7f800000u - kSqrtLo;  // up to infinity
__device__ __forceinline__ float2 sqrt_newton2(const float2 q) {
  float2 y;
  asm("rsqrt.approx.f32 %0, %1;" : "=f"(y.x) : "f"(q.x));
  asm("rsqrt.approx.f32 %0, %1;" : "=f"(y.y) : "f"(q.y));
  const float2 s = __fmul2_rn(q, y), h = __fmul2_rn(both(0.5f), y);
  const float2 r = __ffma2_rn(make_float2(-s.x, -s.y), s, q);
  return __ffma2_rn(r, h, s);
}

__device__ __forceinline__ float sqrt_rn(const float q) {
  if (__float_as_uint(q) - kSqrtLo >= kSqrtSpan) return sqrtf(q);
  float y;
  asm("rsqrt.approx.f32 %0, %1;" : "=f"(y) : "f"(q));
  const float s = __fmul_rn(q, y), h = __fmul_rn(0.5f, y);
  return __fmaf_rn(__fmaf_rn(-s, s, q), h, s);
}

}  // namespace ps2
