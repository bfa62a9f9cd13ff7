// FP64 operations with few instructions on the FP64 pipe, which runs at 1/64
// of the FP32 rate on this part: conversions by integer operations, and a
// quotient and an eighth root by one high-order iteration in FP64 from an
// FP32 estimate.  (A square root made the same way measured slower than
// sqrt().)  The Lagrangian epilogue at 128^3, with its two time scales' roots
// and seven quotients: 3.24 ms a launch in FP64 against 3.44 with the
// functions, 2.03 against 2.22 in the double-word form.
#pragma once
#include <cuda_runtime.h>

namespace lesgo {

// FP32 <-> FP64 by moving exponent and mantissa with integer operations.
// `odd` collects whether a value needs the instruction (zeros, subnormals,
// infinities, NaN; for narrow_fast also results outside the normal range).
__device__ __forceinline__ double widen_fast(float x, bool& odd) {
  const unsigned b = __float_as_uint(x);
  odd |= (b & 0x7f800000u) - 0x00800000u >= 0x7f000000u;   // exponent 0 or 255
  return __hiloint2double((int)(((b & 0x7fffffffu) >> 3) + 0x38000000u | (b & 0x80000000u)), (int)(b << 29));
}
__device__ __forceinline__ float narrow_fast(double x, bool& odd) {   // round to nearest even
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  odd |= (hi & 0x7fffffffu) - 0x38100000u >= 0x0fd00000u;   // outside 2^-126 .. 2^127
  const unsigned l = lo + 0x0fffffffu + ((lo >> 29) & 1u), h = (hi & 0x7fffffffu) + (l < lo ? 1u : 0u);
  return __uint_as_float((__funnelshift_l(l, h, 3) - 0xc0000000u) | (hi & 0x80000000u));
}

// |x| within 2^-100 .. 2^100: the FP32 estimates below are normal numbers
__device__ __forceinline__ bool mid_range(double x) {
  return ((unsigned)__double2hiint(x) & 0x7fffffffu) - 0x39b00000u < 0x0c800000u;
}

// a / b: Newton's iteration for 1 / b from the FP32 reciprocal (2e-7 -> 6e-14)
// and one residual correction of the quotient; within an ulp or so of the
// division, in five FP64 operations.
__device__ __forceinline__ double div_light(double a, double b) {
  bool odd = false;
  const double r0 = widen_fast(__fdividef(1.0f, narrow_fast(b, odd)), odd);
  const double r = fma(r0, fma(-b, r0, 1.0), r0);
  const double q = a * r;
  const double y = fma(fma(-b, q, a), r, q);
  return mid_range(b) && (mid_range(a) || a == 0.0) ? y : a / b;
}
__device__ __forceinline__ float div_light(float a, float b) { return a / b; }

// x^(-1/8), x > 0: Householder's third-order step y (1 + h/8 + 9 h^2/128),
// h = 1 - x y^8, from the FP32 value (the error 0.05 h^3 vanishes in FP64).
__device__ __forceinline__ double inv_root8(double x) {
  bool odd = false;
  const double y = widen_fast(rsqrtf(sqrtf(sqrtf(narrow_fast(x, odd)))), odd);
  const double y2 = y * y, y4 = y2 * y2;
  const double h = fma(-x, y4 * y4, 1.0);
  const double r = fma(y, h * fma(h, 0.0703125, 0.125), y);
  return mid_range(x) && x > 0.0 ? r : rsqrt(sqrt(sqrt(x)));
}
__device__ __forceinline__ float inv_root8(float x) { return rsqrtf(sqrtf(sqrtf(x))); }

}  // namespace lesgo
