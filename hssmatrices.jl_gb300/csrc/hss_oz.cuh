// FP64 products of K <= 128 terms on the 5th-generation tensor cores by the
// error-free splitting of Ozaki, Ogita, Oishi and Rump (2012), with a check
// that sends every output for which the splitting could be less accurate than
// an FP64 sum to that sum.  Shared by the kernels that use it.
//
// Splitting.  A row a of K entries has the exponent E of its largest entry; its
// entries are cut to 63-bit fixed point, a_k = F_k 2^(E - 1085) with E biased and
// |F_k| < 2^63, and F_k cut into nine 7-bit digits, each exact in bf16.  A column
// x likewise (exponent G).  A digit product summed over K <= 128 is an integer
// below 128 * 127^2 < 2^21; the products of one anti-diagonal d = p + q <= 8 add
// up exactly in FP32 (< 2^24: the last digit of an entry is not zero only where
// its first is below 8, so the nine products of d = 8 come to eight at most):
// accumulator d of tensor memory holds S_d = sum_{p + q = d} A_p X_q, and
//     a . x = 2^(E + G - 2114) T,   T = sum_{d <= 8} S_d 2^(56 - 7 d),
// an integer below 2^78 that is put together and rounded once to FP64 by
// integer instructions (GB300 issues FP64 at 1/64 of its FP32 rate).
//
// Check.  With u = 2^(E + G - 2044), above every |a_k x_k|: the cut to fixed
// point and the dropped digit products (d > 8) err by at most
// 10 K 2^-63 u; an FP64 sum of the same terms has the bound K 2^-53 M,
// M = sum |a_k| |x_k|.  The tensor cores also form
// S_abs = sum |top digit of a_k| |top digit of x_k|, and M >= S_abs 2^-14 u, so
// S_abs >= 161 makes the first bound (with the final rounding, at K = 128; 192 at
// K = 6) the smaller one.  Outputs with S_abs below kAbsMin, and rows and
// columns with infinities, NaN, or exponents near the ends of the range, are
// summed in FP64 from the operands instead.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace hss {
namespace oz {

constexpr int kDigits = 9;           // 7-bit digits per value
constexpr int kSlices = kDigits + 1; // and |top digit|, for the check
constexpr int kAcc = 9;              // accumulators S_0 .. S_8; S_abs follows them
constexpr float kAbsMin = 192.f;
constexpr uint32_t kWaitLimit = 1u << 24;

// Exponent codes of a row (column): its largest biased exponent, or one of
constexpr int kZero = -(1 << 28);    // all entries are zero
constexpr int kFar = 1 << 20;        // infinities, NaN, subnormal or nearly so: summed in FP64

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor: no swizzle, K-major 8 x 8 core matrices of
// 128 contiguous bytes, 128 bytes between core matrices along K, 512 along M/N
// (a stage of K = 32), descriptor version 1.
__device__ __forceinline__ uint64_t sdesc(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(512 >> 4) << 32) |
         ((uint64_t)1 << 46);
}
// Byte offset of row (column) i, K group kg (8 entries) in a slice of K = 32.
__device__ __forceinline__ int core_off(int i, int kg) { return (i >> 3) * 512 + kg * 128 + (i & 7) * 16; }

// kind::f16, FP32 accumulator, bf16 K-major operands, M x N.
__host__ __device__ constexpr uint32_t idesc(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mma(uint32_t tmem, uint64_t ad, uint64_t bd, uint32_t id, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
      "l"(ad), "l"(bd), "r"(id), "r"(accumulate));
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)));
}
// Bounded wait for the mbarrier phase `parity`; false when it ran out.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  uint32_t done = 0;
  for (uint32_t it = 0; it < kWaitLimit; ++it) {
    asm volatile(
        "{\n.reg .pred q;\nmbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\nselp.u32 %0, 1, 0, q;\n}\n"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}
// The same with a limit of its own; the first poll does not block, so that a limit of
// one poll can run out.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint32_t limit) {
  uint32_t done;
  asm volatile(
      "{\n.reg .pred q;\nmbarrier.test_wait.parity.shared::cta.b64 q, [%1], %2;\nselp.u32 %0, 1, 0, q;\n}\n"
      : "=r"(done)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  for (uint32_t it = 1; !done && it < limit; ++it)
    asm volatile(
        "{\n.reg .pred q;\nmbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\nselp.u32 %0, 1, 0, q;\n}\n"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
  return done != 0;
}
// Bulk asynchronous copy global -> shared, completion counted on `bar`.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ unsigned long long bits_of(double x) { return (unsigned long long)__double_as_longlong(x); }
__device__ __forceinline__ int biased_exp(unsigned long long b) { return (int)((b >> 52) & 0x7FF); }

// Largest |high word| and the OR of all bits but the signs, over a row's entries.
__device__ __forceinline__ void scan(unsigned long long b, uint32_t& hmax, uint32_t& any) {
  const uint32_t h = (uint32_t)(b >> 32) & 0x7FFFFFFFu;
  hmax = max(hmax, h);
  any |= h | (uint32_t)b;
}

// Exponent code from the largest biased exponent and whether any entry is not zero.
__device__ __forceinline__ int exp_code(int emax, bool any) {
  return !any ? kZero : (emax < 64 || emax == 0x7FF) ? kFar : emax;
}

// |x| cut to 63-bit fixed point relative to biased exponent emax: digits 0..3 and
// 4..7 as 28-bit words, digit 8.  shr.b64 gives 0 for shifts of 64 and more, which
// takes care of zeros and subnormals (rows with a code have emax >= 64).
__device__ __forceinline__ void fixed63(unsigned long long b, int emax, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  const uint32_t bh = (uint32_t)(b >> 32);
  const unsigned long long L = (b << 11) | (1ull << 63);
  const uint32_t sh = (uint32_t)(emax + 1) - ((bh >> 20) & 0x7FFu);
  unsigned long long F;
  asm("shr.b64 %0, %1, %2;" : "=l"(F) : "l"(L), "r"(sh));
  hi = (uint32_t)(F >> 35);
  mid = (uint32_t)(F >> 7) & 0xFFFFFFFu;
  lo = (uint32_t)F & 0x7Fu;
}

// The digits of a pair of values as packed bf16 pairs (first value in the low
// half): a digit a < 128 is the bf16 128 + a (bits 0x4300 | a) minus 128, both
// exact, multiplied by the sign in the same packed FMA.
struct Pair {
  uint32_t h0, m0, h1, m1, l, sg;   // l: the last digits, packed; sg: the signs as a packed pair of +-1
  __device__ __forceinline__ Pair(unsigned long long b0, unsigned long long b1, int emax) {
    uint32_t l0, l1;
    fixed63(b0, emax, h0, m0, l0);
    fixed63(b1, emax, h1, m1, l1);
    l = l0 | (l1 << 16) | 0x43004300u;
    const uint32_t s = ((uint32_t)(b0 >> 63) << 15) | ((uint32_t)(b1 >> 32) & 0x80000000u);
    sg = 0x3F803F80u ^ s;
  }
  __device__ __forceinline__ uint32_t raw(int p) const {   // 128 + digit, both values
    if (p == 8) return l;
    const int s = 21 - 7 * (p & 3);
    const uint32_t a = p < 4 ? h0 : m0, c = p < 4 ? h1 : m1;
    const uint32_t u = s <= 16 ? c << (16 - s) : c >> (s - 16);
    return ((a >> s) & 0x7Fu) | (u & 0x7F0000u) | 0x43004300u;
  }
  __device__ __forceinline__ uint32_t digit(int p) const {
    const uint32_t w = raw(p);
    const uint32_t off = sg ^ 0xFC80FC80u;   // -128 times the signs
    const __nv_bfloat162 v =
        __hfma2(*reinterpret_cast<const __nv_bfloat162*>(&w), *reinterpret_cast<const __nv_bfloat162*>(&sg),
                *reinterpret_cast<const __nv_bfloat162*>(&off));
    return *reinterpret_cast<const uint32_t*>(&v);
  }
  __device__ __forceinline__ uint32_t top_abs() const {
    const uint32_t w = raw(0), m = 0xC300C300u;
    const __nv_bfloat162 v =
        __hadd2(*reinterpret_cast<const __nv_bfloat162*>(&w), *reinterpret_cast<const __nv_bfloat162*>(&m));
    return *reinterpret_cast<const uint32_t*>(&v);
  }
};

// Whether row code ea and column code eb allow the splitting: the sum of the
// exponents keeps the result within FP64's normal range (codes of kFar and
// kZero fall outside).
__device__ __forceinline__ bool in_range(int ea, int eb) { return (unsigned)(ea + eb - 1100) <= 1900u; }
// Both rows are zero-free of contribution: one is all zeros, the other finite.
__device__ __forceinline__ bool is_zero(int ea, int eb) {
  return (ea == kZero && eb != kFar) || (eb == kZero && ea != kFar);
}

// T 2^ex rounded to FP64, T = hi 2^35 + lo (|hi| < 2^44, |lo| < 2^54).
__device__ __forceinline__ double assemble(long long hi, long long lo, int ex) {
  constexpr unsigned long long kLow = (1ull << 35) - 1;
  long long h = hi + (lo >> 35);
  unsigned long long l = (unsigned long long)lo & kLow;
  const bool neg = h < 0;
  if (neg) {
    h = l ? ~h : -h;
    l = (0ull - l) & kLow;
  }
  const int s = min(__clzll(h), 35);
  unsigned long long M = ((unsigned long long)h << s) | (l >> (35 - s));
  const int z = __clzll(M);
  if (z == 64) return 0.0;
  M <<= z;
  const unsigned long long mant = (M >> 11) + ((M >> 10) & 1);
  const int be = 1023 + 63 + 35 - s - z + ex;
  const unsigned long long b = ((unsigned long long)(uint32_t)(be - 1) << 52) + mant;
  return __longlong_as_double((long long)(b | ((unsigned long long)neg << 63)));
}

// Four consecutive 32-bit columns of this warp's tensor-memory lanes.
__device__ __forceinline__ void tmem_ld4(uint32_t addr, float (&v)[4]) {
  uint32_t w[4];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3])
               : "r"(addr));
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = __uint_as_float(w[i]);
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// The four T of columns c .. c + 3 as (hi, lo) and S_abs, from accumulators of
// NC columns each (accumulator d at column NC d, S_abs at NC kAcc).
template <int NC>
__device__ __forceinline__ void gather4(uint32_t tmem, long long (&hi)[4], long long (&lo)[4], float (&sabs)[4]) {
  {
    float v[4][4];
#pragma unroll
    for (int d = 0; d < 4; ++d) tmem_ld4(tmem + (uint32_t)(NC * d), v[d]);
    tmem_wait_ld();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      hi[i] = __float2int_rn(v[3][i]);
#pragma unroll
      for (int d = 0; d < 3; ++d) hi[i] += (long long)__float2int_rn(v[d][i]) * (1 << (21 - 7 * d));
    }
  }
  float v[5][4];
#pragma unroll
  for (int d = 0; d < 5; ++d) tmem_ld4(tmem + (uint32_t)(NC * (d + 4)), v[d]);
  tmem_ld4(tmem + (uint32_t)(NC * kAcc), sabs);
  tmem_wait_ld();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    lo[i] = __float2int_rn(v[4][i]);
#pragma unroll
    for (int d = 0; d < 4; ++d) lo[i] += (long long)__float2int_rn(v[d][i]) * (1 << (28 - 7 * d));
  }
}

// All digit products of one stage (K = 32): slices p of A at a0 + p * astride,
// slices q of X at b0 + q * NC * 64 (so that consecutive q are one operand of
// up to 256 columns), |top| slices behind the digits of each; `first`: the
// accumulators are overwritten.
template <int M, int NC>
__device__ __forceinline__ void stage_mma(uint32_t tmem, uint32_t a0, uint32_t astride, uint32_t b0, bool first) {
  constexpr uint32_t bstride = NC * 64;
#pragma unroll
  for (int kk = 0; kk < 2; ++kk) {
    const bool ow = first && kk == 0;
    // p = 1 reaches S_1 .. S_8 and p = 0 first S_0 alone, so that every
    // accumulator is first written by a product that overwrites it
    mma(tmem + NC, sdesc(a0 + astride + 256 * kk), sdesc(b0 + 256 * kk), idesc(M, 8 * NC), !ow);
    mma(tmem, sdesc(a0 + 256 * kk), sdesc(b0 + 256 * kk), idesc(M, NC), !ow);
    mma(tmem + NC, sdesc(a0 + 256 * kk), sdesc(b0 + bstride + 256 * kk), idesc(M, 8 * NC), 1);
#pragma unroll
    for (int p = 2; p < kDigits; ++p)
      mma(tmem + NC * p, sdesc(a0 + p * astride + 256 * kk), sdesc(b0 + 256 * kk), idesc(M, (9 - p) * NC), 1);
    mma(tmem + NC * kAcc, sdesc(a0 + kDigits * astride + 256 * kk), sdesc(b0 + kDigits * bstride + 256 * kk),
        idesc(M, NC), !ow);
  }
}

}  // namespace oz
}  // namespace hss
