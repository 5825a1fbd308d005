// Reciprocals, quotients and the scalars of a reflector for the factorization and solve
// kernels.  GB300 issues an FP64 warp instruction every 64 clocks per SM sub-partition,
// and a square root or a division is about twenty of them.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace hss {
namespace fac {

__device__ __forceinline__ float fma_t(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fma_t(double a, double b, double c) { return fma(a, b, c); }

// 1 / sqrt(t) and 1 / d for normal t, d > 0 from FP32 seeds (relative error below 2^-21)
// by one step of third order each, the series of (1 - e)^(-1/2) and (1 - e)^(-1) in the
// seed's residual e = 1 - f y^2 (1 - f r) cut after e^2.  A square root and two divisions
// are about forty FP64 instructions on the critical path of every reflector (here 5 and 3).
__device__ __forceinline__ double widen(float x) {   // exact, without an FP64 instruction (x normal)
  const uint32_t b = __float_as_uint(x);
  return __hiloint2double((int)((b >> 3) + (896u << 20)), (int)(b << 29));
}
__device__ __forceinline__ double rsqrt_series(double t) {
  // t = f 4^q with f in [1/2, 2): the seed from f, the power of two put back
  const long long b = __double_as_longlong(t);
  const int q = (int)((b >> 52) - 1022) >> 1;
  const long long fb = b - ((long long)q << 53);
  // f's leading bits as an FP32 number
  const float ff = __uint_as_float((uint32_t)(((fb >> 52) - 1023 + 127) << 23) | (uint32_t)((fb >> 29) & 0x7FFFFF));
  const double f = __longlong_as_double(fb), y = widen(rsqrtf(ff));
  const double e = fma(-f * y, y, 1.0);                      // 1 - f y^2
  const double r = fma(y, e * fma(0.375, e, 0.5), y);
  return __longlong_as_double(__double_as_longlong(r) - ((long long)q << 52));
}
__device__ __forceinline__ double rcp_series(double d) {
  const long long b = __double_as_longlong(d);
  const int q = (int)(b >> 52) - 1023;   // d = f 2^q, f in [1, 2)
  const double f = __longlong_as_double(b - ((long long)q << 52));
  const double r = widen(__frcp_rn(__uint_as_float(0x3F800000u | (uint32_t)((b >> 29) & 0x7FFFFF))));
  const double e = fma(-f, r, 1.0);
  return __longlong_as_double(__double_as_longlong(fma(r, fma(e, e, e), r)) - ((long long)q << 52));
}

__device__ __forceinline__ float recip(float d) { return 1.f / d; }
__device__ __forceinline__ double recip(double d) {
  const int e = (int)(__double_as_longlong(d) >> 52) & 0x7FF;
  if (e < 64 || e > 1982) return 1.0 / d;
  const double r = rcp_series(__longlong_as_double(__double_as_longlong(d) & 0x7FFFFFFFFFFFFFFFll));
  return copysign(r, d);
}

// Tests of the exponent on the bits (FP64 comparisons take the FP64 pipe too).
__device__ __forceinline__ bool is_finite(float x) { return (__float_as_uint(x) & 0x7F800000u) != 0x7F800000u; }
__device__ __forceinline__ bool is_finite(double x) { return (__double2hiint(x) & 0x7FF00000) != 0x7FF00000; }
__device__ __forceinline__ bool is_normal(float x) { return is_finite(x) && (__float_as_uint(x) & 0x7F800000u) != 0; }
__device__ __forceinline__ bool is_normal(double x) { return is_finite(x) && (__double2hiint(x) & 0x7FF00000) != 0; }

// b / d from r = 1 / d: the product and one correction, for a substitution's chain.  It
// is the quotient unless quot_failed says otherwise.
template <typename T>
__device__ __forceinline__ T quot(T b, T d, T r) {
  const T x = b * r;
  return fma_t(r, fma_t(-d, x, b), x);
}
// Whether y = quot(b, d, r) may not be b / d: it is not finite (d zero, infinite or too
// small for its reciprocal, b infinite, a quotient out of range), or b is so small
// (below 2^-118, 2^-1012) that the correction may underflow.
__device__ __forceinline__ bool quot_failed(float y, float d) {
  const uint32_t ey = (__float_as_uint(y) >> 23) & 0xFFu, ed = (__float_as_uint(d) >> 23) & 0xFFu;
  return ey == 0xFFu || ((__float_as_uint(y) << 1) != 0 && ey + ed < 254u - 118u);
}
__device__ __forceinline__ bool quot_failed(double y, double d) {
  const uint32_t ey = ((uint32_t)__double2hiint(y) >> 20) & 0x7FFu, ed = ((uint32_t)__double2hiint(d) >> 20) & 0x7FFu;
  return ey == 0x7FFu || (((unsigned long long)__double_as_longlong(y) << 1) != 0 && ey + ed < 2046u - 1012u);
}

// x / d for several x of at most d's magnitude: by the reciprocal where that is a normal
// number, else by division.
template <typename T>
struct Multiplier {
  T d, r;
  bool fast;
  __device__ __forceinline__ explicit Multiplier(T pivot) : d(pivot), r(recip(pivot)), fast(is_normal(r)) {}
  __device__ __forceinline__ T operator()(T x) const { return fast ? x * r : x / d; }
};

// xLARFG from alpha and the squared tail norm: the norm as sqrt(alpha^2 + ss)
// (hypot only near overflow or underflow); FP32 with correctly rounded
// reciprocals, FP64 with the series above.
__device__ __forceinline__ void larfg_t(float alpha, float ss, float& beta, float& tau, float& scal) {
  if (ss == 0.f) {
    tau = 0.f;
    beta = alpha;
    scal = 1.f;
    return;
  }
  const float t = fmaf(alpha, alpha, ss);
  const float nrm = t <= 3.0e38f ? sqrtf(t) : hypotf(alpha, sqrtf(ss));
  beta = -copysignf(nrm, alpha);
  tau = (beta - alpha) * __frcp_rn(beta);
  scal = __frcp_rn(alpha - beta);
}
__device__ __forceinline__ void larfg_t(double alpha, double ss, double& beta, double& tau, double& scal) {
  // tests on the bits: FP64 comparisons take the FP64 pipe too
  if ((__double_as_longlong(ss) << 1) == 0) {
    tau = 0.0;
    beta = alpha;
    scal = 1.0;
    return;
  }
  const double t = fma(alpha, alpha, ss);
  const int et = (int)(__double_as_longlong(t) >> 52);   // biased exponent (t >= 0)
  if (et > 100 && et < 1946) {
    const double y = rsqrt_series(t), a = fabs(alpha);
    const double nrm = t * y;
    beta = -copysign(nrm, alpha);
    tau = fma(a, y, 1.0);                            // (beta - alpha) / beta
    scal = copysign(rcp_series(a + nrm), alpha);     // 1 / (alpha - beta)
    return;
  }
  const double nrm = hypot(alpha, sqrt(ss));
  beta = -copysign(nrm, alpha);
  tau = (beta - alpha) / beta;
  scal = 1.0 / (alpha - beta);
}

}  // namespace fac
}  // namespace hss
