// FP64 helpers with few FP64 instructions (65 cycles each per warp and sub-partition): comparisons and exponents on the
// integer pipes, reciprocals and square roots by Newton's iteration from an FP32 approximation.
#pragma once

namespace gx {

__device__ __forceinline__ long long dp_bits(double x) { return __double_as_longlong(x); }
__device__ __forceinline__ double dp_abs(double x) { return __hiloint2double(__double2hiint(x) & 0x7fffffff, __double2loint(x)); }
// the larger of two numbers of which at most one is negative; as fmax, a number before a NaN
__device__ __forceinline__ double dp_max(double a, double b) {
  const long long x = dp_bits(a), y = dp_bits(b), inf = 0x7ff0000000000000ll;
  return (x > y && x <= inf) || y > inf ? a : b;
}
// x >= 0 and x <= 0 (signed zeros aside), false for NaN
__device__ __forceinline__ bool dp_ge0(double x) { return (unsigned)__double2hiint(x) <= 0x7ff00000u; }
__device__ __forceinline__ bool dp_le0(double x) {
  const unsigned h = (unsigned)__double2hiint(x);
  return h >= 0x80000000u && h <= 0xfff00000u;
}
// x * 2^k where neither leaves the normal range
__device__ __forceinline__ double dp_scale(double x, int k) { return __hiloint2double(__double2hiint(x) + (k << 20), __double2loint(x)); }
// a positive float in [2^-126, 2^127] times 2^k as a double, by integer instructions
__device__ __forceinline__ double dp_widen(float f, int k) {
  const int b = __float_as_int(f);
  return __hiloint2double((((b >> 23) + 1023 - 127 + k) << 20) | ((b & 0x7fffff) >> 3), b << 29);
}
// Outside the exponents for which the FP32 approximations and the remainders below are normal numbers (zeros,
// subnormal and huge numbers, infinities, NaN) the helpers return what CUDA's operators return.
static __device__ __noinline__ double dp_rcp_rare(double x) { return 1. / x; }
static __device__ __noinline__ double dp_div_rare(double a, double b) { return a / b; }
static __device__ __noinline__ double dp_rsqrt_rare(double x) { return 1. / sqrt(x); }
static __device__ __noinline__ double dp_sqrt_rare(double x) { return sqrt(x); }
// biased exponent e0 .. e0 + count - 1 (sign aside)
__device__ __forceinline__ bool dp_exponent_in(double x, int e0, int count) {
  return (unsigned)(((__double2hiint(x) >> 20) & 0x7ff) - e0) < (unsigned)count;
}

// 1/x: Newton-Raphson r <- r + r (1 - x r) from the 22-bit FP32 approximation of the mantissa's reciprocal.  The
// last step's correction is exact to 2^-33 ulp, so the result is the rounded quotient or, next to a tie, its
// neighbour.
__device__ __forceinline__ double dp_rcp(double x) {
  const int hi = __double2hiint(x), e = (hi >> 20) & 0x7ff;
  if (!dp_exponent_in(x, 123, 1800)) return dp_rcp_rare(x);
  const float m = __int_as_float(0x3f800000 | ((hi & 0xfffff) << 3) | (int)((unsigned)__double2loint(x) >> 29));
  double r = dp_widen(__fdividef(1.f, m), 1023 - e);
  r = __hiloint2double(__double2hiint(r) | (hi & 0x80000000), __double2loint(r));
  r = fma(r, fma(-x, r, 1.), r);
  return fma(r, fma(-x, r, 1.), r);
}
// a/b with the remainder of the first quotient (as close to the rounded quotient as dp_rcp); both within
// 2^-500 .. 2^500, where quotient and remainder are normal numbers
__device__ __forceinline__ double dp_div(double a, double b) {
  if (!dp_exponent_in(a, 523, 1000) || !dp_exponent_in(b, 523, 1000)) return dp_div_rare(a, b);
  const double r = dp_rcp(b), q = a * r;
  return fma(fma(-b, q, a), r, q);
}
// y = 1/sqrt(x) by Newton's iteration y <- y + y/2 (1 - x y y) from the FP32 approximation, to one ulp (the rounding
// of x y), and sqrt(x): with the remainder of x y (EXACT) or x y itself, to two ulp
template <bool EXACT>
__device__ __forceinline__ double dp_root(double x, double& y) {
  const int hi = __double2hiint(x);
  if ((unsigned)((hi >> 20) - 123) >= 1800u) {  // also every negative x
    y = dp_rsqrt_rare(x);
    return dp_sqrt_rare(x);
  }
  const int e = (hi >> 20) - 1023, k = e >> 1;  // x = m 2^(2k), 1 <= m < 4
  const float m = __int_as_float(((127 + (e - 2 * k)) << 23) | ((hi & 0xfffff) << 3) | (int)((unsigned)__double2loint(x) >> 29));
  y = dp_widen(rsqrtf(m), -k);
  y = fma(dp_scale(y, -1), fma(-(x * y), y, 1.), y);
  y = fma(dp_scale(y, -1), fma(-(x * y), y, 1.), y);
  const double s = x * y;
  return EXACT ? fma(fma(-s, s, x), dp_scale(y, -1), s) : s;
}
__device__ __forceinline__ double dp_sqrt(double x) {
  double y;
  return dp_root<true>(x, y);
}

}  // namespace gx
