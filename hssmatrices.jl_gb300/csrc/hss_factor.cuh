// Device pieces shared by the two ULV factorization kernels (hss_factor_blk.cu,
// hss_factor_pan.cu): 256 threads per block, panels of 32 reflectors with 8
// lanes per column (QL) or row (LQ).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "hss_device.cuh"
#include "hss_internal.h"

namespace hss {
namespace fac {

constexpr int NT = 256;             // threads per block
constexpr int NW = NT / 32;
constexpr int BP = 32;              // panel width (reflectors per panel)
constexpr int PL = 8;               // lanes per panel column (QL) or row (LQ)
constexpr int GP = BP + 1;          // ld of the Gram matrix and of T
static_assert(NT == 8 * BP, "the panel mapping puts 8 lanes on each of 32 columns (rows)");

__device__ __forceinline__ float fma_t(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fma_t(double a, double b, double c) { return fma(a, b, c); }

template <typename T>
__device__ __forceinline__ T gsum8(T v, unsigned gm) {   // sum over the 8 lanes of a group
  v += __shfl_xor_sync(gm, v, 4);
  v += __shfl_xor_sync(gm, v, 2);
  v += __shfl_xor_sync(gm, v, 1);
  return v;
}

// xLARFG from alpha and the squared tail norm: the norm as sqrt(alpha^2 + ss)
// (hypot only near overflow or underflow); FP32 with correctly rounded
// reciprocals, FP64 with the Newton steps above.
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
// 1 / sqrt(t) and 1 / d for normal t, d > 0 from FP32 seeds (relative error e below
// 2^-21) by one step of third order each: GB300 issues an FP64 warp instruction
// every 64 clocks per SM sub-partition, and a square root and two divisions are
// about forty of them on the critical path of every reflector (here 5 and 3).
__device__ __forceinline__ double widen(float x) {   // exact, without an FP64 instruction (x normal)
  const uint32_t b = __float_as_uint(x);
  return __hiloint2double((int)((b >> 3) + (896u << 20)), (int)(b << 29));
}
__device__ __forceinline__ double rsqrt_newton(double t) {
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
__device__ __forceinline__ double rcp_newton(double d) {
  const long long b = __double_as_longlong(d);
  const int q = (int)(b >> 52) - 1023;   // d = f 2^q, f in [1, 2)
  const double f = __longlong_as_double(b - ((long long)q << 52));
  const double r = widen(__frcp_rn(__uint_as_float(0x3F800000u | (uint32_t)((b >> 29) & 0x7FFFFF))));
  const double e = fma(-f, r, 1.0);
  return __longlong_as_double(__double_as_longlong(fma(r, fma(e, e, e), r)) - ((long long)q << 52));
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
    const double y = rsqrt_newton(t), a = fabs(alpha);
    const double nrm = t * y;
    beta = -copysign(nrm, alpha);
    tau = fma(a, y, 1.0);                            // (beta - alpha) / beta
    scal = copysign(rcp_newton(a + nrm), alpha);     // 1 / (alpha - beta)
    return;
  }
  const double nrm = hypot(alpha, sqrt(ss));
  beta = -copysign(nrm, alpha);
  tau = (beta - alpha) / beta;
  scal = 1.0 / (alpha - beta);
}

// four consecutive elements, 16-byte aligned (FP32) or 32-byte aligned (FP64)
__device__ __forceinline__ void ld4(float (&v)[4], const float* p) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}
__device__ __forceinline__ void ld4(double (&v)[4], const double* p) {
  const double2 a = reinterpret_cast<const double2*>(p)[0];
  const double2 b = reinterpret_cast<const double2*>(p)[1];
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}

// acc += a . b over four entries as a chain of fused multiply-adds
template <typename T>
__device__ __forceinline__ void fma4(T& acc, const T (&a)[4], const T (&b)[4]) {
  acc = fma_t(a[0], b[0], acc);
  acc = fma_t(a[1], b[1], acc);
  acc = fma_t(a[2], b[2], acc);
  acc = fma_t(a[3], b[3], acc);
}

// LU with partial pivoting of an m x m block in shared memory (ld).
template <typename T>
__device__ void lu_blk(T* A, int m, int ld, int32_t* piv, int32_t* err, T* bv, int* bi, int* prow) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int c = 0; c < m; ++c) {
    T best = T(-1);
    int idx = m;
    for (int i = c + tid; i < m; i += NT) {
      const T a = dabs(A[i + c * ld]);
      if (a > best) { best = a; idx = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const T ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
      if (ob > best || (ob == best && oi < idx)) { best = ob; idx = oi; }
    }
    if (lane == 0) { bv[warp] = best; bi[warp] = idx; }
    __syncthreads();
    if (tid == 0) {
      T b = bv[0];
      int ix = bi[0];
      for (int w = 1; w < NW; ++w)
        if (bv[w] > b || (bv[w] == b && bi[w] < ix)) { b = bv[w]; ix = bi[w]; }
      if (ix >= m) ix = c;
      *prow = ix;
      piv[c] = ix;
      if (A[ix + c * ld] == T(0) && err != nullptr) atomicExch(err, DEV_SINGULAR);
    }
    __syncthreads();
    const int p = *prow;
    if (p != c)
      for (int j = tid; j < m; j += NT) {
        const T t = A[c + j * ld];
        A[c + j * ld] = A[p + j * ld];
        A[p + j * ld] = t;
      }
    __syncthreads();
    const T d = A[c + c * ld];
    if (d != T(0))
      for (int i = c + 1 + tid; i < m; i += NT) A[i + c * ld] /= d;
    __syncthreads();
    const int rem = m - c - 1;
    for (int e = tid; e < rem * rem; e += NT) {
      const int i = c + 1 + e % rem, j = c + 1 + e / rem;
      A[i + j * ld] -= A[i + c * ld] * A[c + j * ld];
    }
    __syncthreads();
  }
}

// T = S^{-1} (S = diag(1/tau) + strictly upper G) by warp 0, one row of T per
// lane in registers, columns in order (xLARFT's recurrence T(i,i) = tau_i,
// T(0:i, i) = -tau_i T(0:i, 0:i) G(0:i, i)).  Tm row-major (ld GP, zero
// outside the upper triangle), also written column-major to Tg (32 x 32).
template <typename T>
__device__ void blk_tmat(int nb, const T* G, const T* tau, T* Tm, T* Tg) {
  if (threadIdx.x < 32) {
    const int l = threadIdx.x;
    T tr[BP];
#pragma unroll
    for (int q = 0; q < BP; ++q) tr[q] = T(0);
#pragma unroll
    for (int i = 0; i < BP; ++i) {
      if (i < nb) {   // warp-uniform
        T s0 = T(0), s1 = T(0);
#pragma unroll
        for (int q = 0; q < i; ++q) {
          if (q & 1) s1 += tr[q] * G[q * GP + i];
          else s0 += tr[q] * G[q * GP + i];
        }
        const T ti = tau[i];
        tr[i] = l < i ? -ti * (s0 + s1) : (l == i ? ti : T(0));
      }
    }
#pragma unroll
    for (int q = 0; q < BP; ++q) {
      Tm[l * GP + q] = tr[q];
      Tg[l + q * BP] = tr[q];
    }
  }
  __syncthreads();
}

// The same T (32 x 32) by halves, for FP64: the four 8 x 8 diagonal blocks by a
// warp each (one row per lane), then T12 = -T1 G12 T2 for blocks of 8 and of 16
// by all threads.  One warp alone would issue 496 dependent FP64 instructions.
// G is overwritten; NTH threads, at least 128.
template <int NTH>
__device__ void blk_tmat_halves(int nb, double* G, const double* tau, double* Tm, double* Tg) {
  const int tid = threadIdx.x, warp = tid >> 5, l = tid & 31;
  for (int e = tid; e < BP * BP; e += NTH) Tm[(e >> 5) * GP + (e & 31)] = 0.0;
  __syncthreads();
  if (warp < 4 && l < 8) {
    const int o = 8 * warp;
    double tr[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      double s = 0.0;
#pragma unroll
      for (int q = 0; q < i; ++q) s = fma(tr[q], G[(o + q) * GP + o + i], s);
      const double ti = o + i < nb ? tau[o + i] : 0.0;
      tr[i] = l < i ? -ti * s : (l == i ? ti : 0.0);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) Tm[(o + l) * GP + o + i] = tr[i];
  }
  __syncthreads();
#pragma unroll
  for (int h = 8; h < BP; h *= 2) {
    // blocks (o, o + h) for o = 0, 2 h, ...: W = G12 T2 into G's block, then T12 = -T1 W
    const int cnt = BP / (2 * h) * h * h;
    double w[(BP / 2 * BP / 2 + NTH - 1) / NTH];
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
      for (int z = 0; z < (BP / 2 * BP / 2 + NTH - 1) / NTH; ++z) {
        const int e = tid + z * NTH;
        if (e < cnt) {
          const int o = e / (h * h) * 2 * h, i = o + e / h % h, j = o + h + e % h;
          double s = 0.0;
          if (pass == 0) {
            for (int q = o + h; q <= j; ++q) s = fma(G[i * GP + q], Tm[q * GP + j], s);
          } else {
            for (int q = i; q < o + h; ++q) s = fma(Tm[i * GP + q], G[q * GP + j], s);
            s = -s;
          }
          w[z] = s;
        }
      }
      __syncthreads();
#pragma unroll
      for (int z = 0; z < (BP / 2 * BP / 2 + NTH - 1) / NTH; ++z) {
        const int e = tid + z * NTH;
        if (e < cnt) {
          const int o = e / (h * h) * 2 * h, i = o + e / h % h, j = o + h + e % h;
          (pass == 0 ? G : Tm)[i * GP + j] = w[z];
        }
      }
      __syncthreads();
    }
  }
  for (int e = tid; e < BP * BP; e += NTH) Tg[e] = Tm[(e & 31) * GP + (e >> 5)];   // Tg column-major
}

}  // namespace fac
}  // namespace hss
