// hss_recip.cuh on the CPU: reciprocals, quotients and reflector scalars against extended
// precision, over the whole range and at its ends (zero, subnormal, huge, infinite, NaN).
// The device's approximate seed rsqrtf is stood in for by the true value moved by up to
// its documented 2 ulp.  Bounds, from the steps' roundings: FP64 reciprocals, square roots
// and quotients 2^-52 relative (two roundings and what the third-order step leaves,
// below 2^-60), reflector scalars 2^-50 (up to eight), FP32 quotients 2^-23; below
// the normal range twice the smallest number.  Quotients give a quotient's infinities, zeros and
// NaN.  Prints one line per failure.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
#include <vector>

static int seed_shift = 0;
template <class A, class B>
static A bits_as(B b) {
  static_assert(sizeof(A) == sizeof(B), "");
  A a;
  std::memcpy(&a, &b, sizeof(a));
  return a;
}
static inline uint32_t __float_as_uint(float x) { return bits_as<uint32_t>(x); }
static inline float __uint_as_float(uint32_t x) { return bits_as<float>(x); }
static inline long long __double_as_longlong(double x) { return bits_as<long long>(x); }
static inline double __longlong_as_double(long long x) { return bits_as<double>(x); }
static inline double __hiloint2double(int hi, int lo) {
  return bits_as<double>(((uint64_t)(uint32_t)hi << 32) | (uint32_t)lo);
}
static inline int __double2hiint(double x) { return (int)(bits_as<uint64_t>(x) >> 32); }
static inline float __frcp_rn(float x) { return 1.f / x; }
static inline float seed_rsqrtf(float x) {
  return bits_as<float>(bits_as<uint32_t>((float)(1.0 / std::sqrt((double)x))) + seed_shift);
}
#define rsqrtf seed_rsqrtf
using std::copysign;
#include "hss_recip.cuh"

using namespace hss::fac;
typedef long double Q;

static int bad = 0;
#define REPORT(...)            \
  do {                         \
    if (++bad < 20) std::printf(__VA_ARGS__); \
  } while (0)

template <class T>
static void check(const char* what, double a, double b, T got, Q want, Q rel) {
  const Q tiny = std::numeric_limits<T>::denorm_min();
  const Q err = std::fabs((Q)got - want), bound = std::fabs(want) * rel;
  const bool sub = std::fabs(want) < 4 * (Q)std::numeric_limits<T>::min();
  if (!(err <= bound || (sub && err <= 2 * tiny))) REPORT("%s(%a, %a) = %a\n", what, a, b, (double)got);
}

template <class T>
static void check_quot(T b, T d, Q rel) {
  const T fast = quot(b, d, recip(d)), div = b / d, got = quot_failed(fast, d) ? div : fast;
  if (std::isnan(div) ? !std::isnan(got) : (std::isinf(div) || std::isinf(got)) ? got != div : false)
    // (a result that rounds up to infinity may be the largest number, and the other way round)
    if (!(std::isfinite(got) != std::isfinite(div) && !std::isnan(got) && b != 0 && d != 0 && std::isfinite(b) &&
          std::fabs((Q)b / d) > (Q)std::numeric_limits<T>::max() * (1 - rel)))
      REPORT("quot(%a, %a) = %a, not %a\n", (double)b, (double)d, (double)got, (double)div);
  if (std::isfinite(div) && std::isfinite(got)) check("quot", b, d, got, (Q)b / (Q)d, rel);
}

int main() {
  const Q u = std::ldexp((Q)1, -53);
  std::mt19937_64 gen(5);
  auto mant = [&]() { return 1.0 + std::ldexp((double)(gen() >> 12), -52); };
  for (seed_shift = -2; seed_shift <= 2; ++seed_shift)
    for (int i = 0; i < 100000; ++i) {
      const int e = (int)(gen() % 1840) - 920;
      const double t = std::ldexp(i < 4 ? 1.0 + (i & 1 ? std::ldexp(1.0, -52) : 0.0) : mant(), e);
      check("rsqrt_series", t, 0, rsqrt_series(t), 1 / std::sqrt((Q)t), 2 * u);
      check("rcp_series", t, 0, rcp_series(t), 1 / (Q)t, 2 * u);
      // a reflector of norm sqrt(alpha^2 + ss), with any share of alpha in it
      const double ss = std::ldexp(mant(), 2 * (e / 2)), al = (gen() & 1 ? 1 : -1) * std::ldexp(mant(), e / 2 + (int)(gen() % 60) - 40);
      double beta, tau, scal;
      larfg_t(al, ss, beta, tau, scal);
      const Q nrm = std::sqrt((Q)al * al + ss), be = al < 0 ? nrm : -nrm;
      check("larfg beta", al, ss, beta, be, 8 * u);
      check("larfg tau", al, ss, tau, (be - al) / be, 8 * u);
      check("larfg scal", al, ss, scal, 1 / (al - be), 8 * u);
    }
  seed_shift = 0;
  for (int i = 0; i < 300000; ++i) {
    const double d = (gen() & 1 ? 1 : -1) * std::ldexp(mant(), (int)(gen() % 2045) - 1022);
    check("recip", d, 0, recip(d), 1 / (Q)d, 2 * u);
    check_quot<double>((gen() & 1 ? 1 : -1) * std::ldexp(mant(), (int)(gen() % 2097) - 1073), d, 2 * u);
    const float df = (float)((gen() & 1 ? 1 : -1) * std::ldexp(mant(), (int)(gen() % 253) - 126));
    check_quot<float>((float)std::ldexp(mant(), (int)(gen() % 276) - 149), df, std::ldexp((Q)1, -23));
  }
  const double in = std::numeric_limits<double>::infinity(), nan = std::numeric_limits<double>::quiet_NaN();
  const std::vector<double> v64{0.0, 1.0, 3.0, 1e-300, 1e300, 1.7e308, 4.9e-324, 1e-310, 2.2250738585072014e-308,
                                1.1125369292536007e-308, 5e307, in, nan};
  const std::vector<double> v32{0.0, 1.0, 3.0, 1e-37, 1e37, 3.4e38, 1.4e-45, 1e-40, 1.1754943508222875e-38, 2.9e-39, 2e38, in, nan};
  for (int s = 0; s < 4; ++s) {
    const double sb = s & 1 ? -1 : 1, sd = s & 2 ? -1 : 1;
    for (double b : v64)
      for (double d : v64) check_quot<double>(sb * b, sd * d, 2 * u);
    for (double b : v32)
      for (double d : v32) check_quot<float>((float)(sb * b), (float)(sd * d), std::ldexp((Q)1, -23));
  }
  // the multipliers of an elimination: x / d for |x| <= |d|
  for (double d : {1.4e-45, 1e-40, 2.9e-39, 1.2e-38, 1.0, 2e38, 3.4e38})
    for (double f : {1.0, 0.5, 0.3}) {
      const float p = (float)d, x = (float)(f * d);
      const Multiplier<float> m(p);
      check("multiplier", x, p, m(x), (Q)x / p, std::ldexp((Q)1, -22));
    }
  for (double d : {4.9e-324, 1e-310, 1.2e-308, 1.0, 1e308, 1.7e308})
    for (double f : {1.0, 0.5, 0.3}) {
      const double x = f * d;
      const Multiplier<double> m(d);
      check("multiplier", x, d, m(x), (Q)x / d, 4 * u);
    }
  if (bad) std::printf("%d failures\n", bad);
  return 0;
}
