// FP64 reciprocals and reciprocal square roots for serial chains: an FP32 estimate and one step of
// third order (Householder's iteration: with e = 1 - d y^2, y (1 + e/2 + 3 e^2 / 8); with e = 1 - x y,
// y (1 + e + e^2); e < 2^-20, so the step's own error is below 2^-60).  Three to six FP64 instructions of
// 64 clocks of an SM quarter each; a division takes 565 and a square root 700.  The last bit may
// differ from the correctly rounded value, and a product with a reciprocal has one rounding more than
// the division.  The solvers that use them show no loss: the errors against 128-bit sums of
// eigenvalues, residuals and harmonic-Ritz residuals are 0.94 to 1.05 times those of the variants with
// divisions (means over 40 to 150 problems, m = 20 to 124), the orthogonality of the vectors 0.6 to
// 1.3 times (set by the gaps), of the Cholesky QR 0.94 to 0.98 times; the Cholesky inverse is off by
// 3.2e-16 to 4.7e-16 of its norm, 3.8e-16 to 4.6e-16 with divisions (n = 64 to 200).
#pragma once

#include "common.cuh"

namespace vgb {

// The float nearest below a double in FP32's range and back, in integers (a conversion is an FP64
// instruction).
__device__ __forceinline__ float to_float(double x) {
  const unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x);
  return __uint_as_float((h & 0x80000000u) | (((h & 0x7FFFFFFFu) - (896u << 20)) << 3) | (l >> 29));
}
__device__ __forceinline__ double to_double(float x) {  // normal x
  const unsigned b = __float_as_uint(x);
  return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7FFFFFFFu) >> 3) + (896u << 20))), (int)(b << 29));
}
// 1 / sqrt(x) and 1 / x for x within [1, 64) from the FP32 estimate f
__device__ __forceinline__ double fast_rsqrt(double x, float f) {
  const double y = to_double(f);
  const double e = fma(-(x * y), y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}
__device__ __forceinline__ double fast_rcp(double x, float f) {
  const double y = to_double(f);
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}
__device__ __forceinline__ double with_sign(double a, double b) {  // |a| with b's sign bit
  return __hiloint2double((__double2hiint(a) & 0x7FFFFFFF) | (__double2hiint(b) & (int)0x80000000), __double2loint(a));
}

// 1 / sqrt(d) for any d > 0 (zeros, infinities and NaN as 1 / sqrt(d) gives them)
__device__ __forceinline__ double rsqrt64(double d) {
  const int h = __double2hiint(d), ex = ((h >> 20) & 0x7FF) - 1023;
  if (h < 0 || ex == -1023 || ex == 1024) return 1.0 / sqrt(d);
  const double m = __hiloint2double((h & 0xFFFFF) | ((1023 + (ex & 1)) << 20), __double2loint(d));  // d = m 4^(ex >> 1)
  float f;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(f) : "f"(to_float(m)));
  const double r = fast_rsqrt(m, f);
  return __hiloint2double(__double2hiint(r) - ((ex >> 1) << 20), __double2loint(r));
}
// 1 / x for any x
__device__ __forceinline__ double rcp64(double x) {
  const int h = __double2hiint(x), ex = ((h >> 20) & 0x7FF) - 1023;
  if (ex < -1000 || ex > 1000) return 1.0 / x;
  const double m = __hiloint2double((h & 0xFFFFF) | (1023 << 20), __double2loint(x));
  float f;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(f) : "f"(to_float(m)));
  const double r = fast_rcp(m, f);
  return __hiloint2double((__double2hiint(r) - (ex << 20)) | (h & (int)0x80000000), __double2loint(r));
}

}  // namespace vgb
