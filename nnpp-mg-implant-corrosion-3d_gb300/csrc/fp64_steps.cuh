// fp64_steps.cuh -- FP64 quotients and reciprocal square roots in fewer FP64 instructions than the
// operators', for chains and bond loops that the FP64 pipe bounds (a warp-wide FP64 instruction holds it
// for 64 cycles).  Published iterations (Newton-Raphson's, Householder's of third order) from a
// single-precision start; tests/test_gpu_fp64_steps.py holds each to 2 units in the last place of the exact
// value over the exponents, and to CUDA's results for zero, subnormal, infinite and NaN operands as
// stated here.
#ifndef NNPP_FP64_STEPS_CUH
#define NNPP_FP64_STEPS_CUH

namespace nnpp {

// the exponent field
__device__ __forceinline__ int exponent_of(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }

// a / b by Newton steps on the reciprocal of b's significand and one correction of the quotient by its
// remainder.  The operator: b zero, subnormal, infinite, NaN or above 2^1022; a below 2^-959 (its remainder
// would be subnormal), zero, infinite or NaN.
__device__ __forceinline__ double div_newton(double a, double b) {
  const int ex = exponent_of(b), ea = exponent_of(a);
  if (ex == 0 || ex >= 0x7fe || ea < 64 || ea == 0x7ff) return a / b;
  const double m = __longlong_as_double((__double_as_longlong(b) & (long long)0x800fffffffffffffull) | 0x3ff0000000000000ll);
  double x = (double)(1.0f / (float)m);
  x = fma(x, fma(-m, x, 1.0), x);
  x = fma(x, fma(-m, x, 1.0), x);
  double q = a * x;
  q = fma(fma(-m, q, a), x, q);
  return q * __longlong_as_double((long long)(2046 - ex) << 52);
}

// a / d from rd = 1 / d (d and rd within 10^+-150) and one correction by the remainder.  The product
// itself where it is infinite or NaN or a is zero, the operator for other a below 2^-959.
__device__ __forceinline__ double div_corrected(double a, double d, double rd) {
  const double q = __dmul_rn(a, rd);
  if (exponent_of(q) == 0x7ff) return q;
  if (exponent_of(a) < 64) return (__double_as_longlong(a) << 1) == 0 ? q : __ddiv_rn(a, d);
  return fma(fma(-q, d, a), rd, q);
}

// 1 / sqrt(x), x > 0: two Newton steps from the FP32 root of x scaled by a power of four into [1, 4);
// subnormal, infinite and NaN x: the operators
__device__ __forceinline__ double rsqrt_newton(double x) {
  const long long bits = __double_as_longlong(x);
  const int ex = (int)(bits >> 52);
  if (ex == 0 || ex >= 0x7ff) return 1.0 / sqrt(x);
  const int odd = (ex + 1) & 1;  // x = m 2^(ex - 1023 - odd), an even power
  const double m = __longlong_as_double((bits & 0x000fffffffffffffll) | (long long)(1023 + odd) << 52);
  double y = (double)rsqrtf((float)m);
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const double r = fma(-m * y, y, 1.0);
    y = fma(0.5 * y, r, y);
  }
  return y * __longlong_as_double((long long)(1023 - (ex - 1023 - odd) / 2) << 52);
}

// 1 / sqrt(x) from a single-precision start y0 (22 bits) and Householder's third-order step
// y0 + y0 e (1/2 + 3/8 e), e = 1 - x y0^2: the error falls to e^3 and stays at the FP64 rounding.
// The conversions move bits, so that only the step's five operations use the FP64 pipe; values
// outside 2^+-100 (zero, infinity, NaN and negative ones among them) take CUDA's rsqrt.
__device__ __forceinline__ double rsqrt_step(double x) {
  const unsigned int hi = (unsigned int)__double2hiint(x), lo = (unsigned int)__double2loint(x);
  const unsigned int ex = hi >> 20;
  if (ex < 1023u - 100u || ex > 1023u + 100u) return rsqrt(x);
  const float f = __uint_as_float(((ex - 1023u + 127u) << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29));
  const unsigned int g = __float_as_uint(rsqrtf(f));
  const double y = __hiloint2double((int)((((g >> 23) - 127u + 1023u) << 20) | ((g & 0x7fffffu) >> 3)), (int)(g << 29));
  const double e = fma(-__dmul_rn(x, y), y, 1.0);
  return fma(__dmul_rn(e, fma(e, 0.375, 0.5)), y, y);
}

}  // namespace nnpp

#endif  // NNPP_FP64_STEPS_CUH
