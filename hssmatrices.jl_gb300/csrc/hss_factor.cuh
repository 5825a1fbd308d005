// Device pieces shared by the two ULV factorization kernels (hss_factor_blk.cu,
// hss_factor_pan.cu): 256 threads per block, panels of 32 reflectors with 8
// lanes per column (QL) or row (LQ).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "hss_device.cuh"
#include "hss_internal.h"
#include "hss_recip.cuh"

namespace hss {
namespace fac {

constexpr int NT = 256;             // threads per block
constexpr int NW = NT / 32;
constexpr int BP = 32;              // panel width (reflectors per panel)
constexpr int PL = 8;               // lanes per panel column (QL) or row (LQ)
constexpr int GP = BP + 1;          // ld of the Gram matrix and of T
static_assert(NT == 8 * BP, "the panel mapping puts 8 lanes on each of 32 columns (rows)");

template <typename T>
__device__ __forceinline__ T gsum8(T v, unsigned gm) {   // sum over the 8 lanes of a group
  v += __shfl_xor_sync(gm, v, 4);
  v += __shfl_xor_sync(gm, v, 2);
  v += __shfl_xor_sync(gm, v, 1);
  return v;
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

// Index of the warp's largest magnitude (ties: the smallest index), by integer
// reductions on the bits; lanes without an entry pass idx >= 2^30.
__device__ __forceinline__ int warp_argmax(float x, int idx, bool& zero) {
  const unsigned a = __float_as_uint(x) & 0x7FFFFFFFu;
  const unsigned best = __reduce_max_sync(0xffffffffu, a);
  zero = best == 0;
  return (int)__reduce_min_sync(0xffffffffu, a == best ? (unsigned)idx : 1u << 30);
}
__device__ __forceinline__ int warp_argmax(double x, int idx, bool& zero) {
  const unsigned long long a = (unsigned long long)__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFull;
  const unsigned hi = (unsigned)(a >> 32), bh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned lo = hi == bh ? (unsigned)a : 0u, bl = __reduce_max_sync(0xffffffffu, lo);
  zero = bh == 0 && bl == 0;
  return (int)__reduce_min_sync(0xffffffffu, hi == bh && lo == bl ? (unsigned)idx : 1u << 30);
}
__device__ __forceinline__ bool larger_mag(float a, float b) {
  return (__float_as_uint(a) & 0x7FFFFFFFu) > (__float_as_uint(b) & 0x7FFFFFFFu);
}
__device__ __forceinline__ bool larger_mag(double a, double b) {
  return ((unsigned long long)__double_as_longlong(a) << 1) > ((unsigned long long)__double_as_longlong(b) << 1);
}
// LU with partial pivoting of an m x m block (ld), columns dealt to the warps in
// turn.  One barrier per column: while the other warps apply column c, the owner
// of column c + 1 applies it there first, finds the next pivot (first entry of
// largest magnitude, compared on the bits: NaN counts as larger than any number)
// and scales that column.  lv: 2 x m multipliers; pv: 2 pivots.  A root of 64 rows
// with its assembly: FP64 215 -> 141 us (five barriers a column, FP64 comparisons
// and a division per entry before), FP32 unchanged at 94; 32 rows 100 -> 55 and
// 39 -> 35 us.
template <typename T>
__device__ void lu_blk(T* A, int m, int ld, int32_t* piv, int32_t* err, T* lv, int* pv) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // pivot and multipliers of column c, by the warp that owns it
  auto next = [&](int c) {
    T* col = A + (int64_t)c * ld;
    T mine = T(0);
    int at = 1 << 30;
    for (int i = c + lane; i < m; i += 32)
      if (at == 1 << 30 || larger_mag(col[i], mine)) { mine = col[i]; at = i; }
    bool zero;
    const int idx = warp_argmax(mine, at, zero);
    if (lane == 0) {
      piv[c] = idx;
      pv[c & 1] = idx;
      if (zero && err != nullptr) atomicExch(err, DEV_SINGULAR);
      const T t = col[c];
      col[c] = col[idx];
      col[idx] = t;
    }
    __syncwarp();
    const Multiplier<T> mult(zero ? T(1) : col[c]);
    T* l = lv + (c & 1) * m;
    for (int i = c + 1 + lane; i < m; i += 32) {
      const T x = mult(col[i]);
      col[i] = x;
      l[i] = x;
    }
    __syncwarp();
  };
  if (m > 0 && warp == 0) next(0);
  __syncthreads();
  for (int c = 0; c < m; ++c) {
    const int p = pv[c & 1];
    const T* l = lv + (c & 1) * m;
    // this warp's columns, the next one first (its owner's first column is c + 1)
    const int first = c + 1 + (warp + NW - (c + 1) % NW) % NW;
    for (int q = 0; q * NW < m; ++q) {
      const int j = (first + q * NW) < m ? first + q * NW : -1;
      if (j < 0) break;
      T* col = A + (int64_t)j * ld;
      const T u = col[p];
      __syncwarp();
      if (lane == 0 && p != c) {
        col[p] = col[c];
        col[c] = u;
      }
      __syncwarp();
      for (int i = c + 1 + lane; i < m; i += 32) col[i] = fma_t(-l[i], u, col[i]);
      __syncwarp();
      if (j == c + 1) next(c + 1);
    }
    // rows already eliminated: exchanged only
    if (p != c)
      for (int j = threadIdx.x; j < c; j += NT) {
        T* col = A + (int64_t)j * ld;
        const T t = col[c];
        col[c] = col[p];
        col[p] = t;
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
