// ULV reduction of one tree level by panels, FP32 or FP64 (restated from
// src/ulvfactor.jl:22-57, the leaf reduction, and :74-79, the merge, with the
// reference's reflector order), the block updates on the tensor cores.
//
// A level is a short sequence of launches over all its nodes, working in the
// factor storage:
//   leaf_copy / merge   D, U, V of the leaves, or assembled from the children;
//   per QL panel        panel_kernel: 32 columns of U reduced (geqlf!, :39), T;
//                       apply_kernel: the panel's I - Y T Y^T on D and the columns
//                       of U to its left (ormql!, :41);
//   per LQ panel        panel_kernel: 32 rows of D[0:mk, :] reduced (gelqf!, :44), T;
//                       apply_kernel: on the rows of D below and on V (ormlq!, :47, :50);
//   root_kernel         the root's LU (:83).
// The factor storage is that of ulv_factor_blk_kernel (without the inverses of L1's
// diagonal blocks, which only its own solve reads), for nodes of any rank and up to
// 512 rows.
//
// Why so: in one block per node the updates are FP64 multiply-adds at 2 per
// clock and SM (2.9 of a leaf's 4 M at 128 x 128, k = 32) or, in FP32, one wave
// after another of blocks that fill an SM's shared memory.  The updates are
// matrix products, S <- S - ((S Y^T) T) Y over a node's rows (columns of D and U
// for QL), so they run as exact bf16 digit products (hss_oz.cuh; FP32 data by
// five digits), which leaves the panels: their blocks are small, so several
// share an SM.
//
// Measured (one GB300): FP64, n = 65536, 512 leaves of 128, k = 32: leaf level 7.3 ->
// 2.8 ms (four panels of 0.41 ms: the FP64 pipe; four updates of 0.18 to 0.45 ms:
// integer instructions of cutting and putting together), a merge level of 64 x 64
// nodes 562 -> 300 us (two panels of 94 us, a chain of 32 reflectors of about 2.2 us;
// two updates of 54 us; the products of the merge 28 us).  FP32, 128 leaves of 156,
// k = 40: 1.47 -> 0.63 ms.  Errors of FP64 solves against a 64-bit elimination are
// 0.8 of those of the updates on the FP64 pipe.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "hss_device.cuh"
#include "hss_factor.cuh"
#include "hss_internal.h"
#include "hss_launch.h"
#include "hss_optin.h"
#include "hss_oz.cuh"

namespace hss {

using namespace fac;

namespace {

constexpr int AT = 512;    // threads of apply_kernel
constexpr int TR = 128;    // rows per block there
constexpr int NCA = 32;    // columns of its products
constexpr int AS = TR * 32 * 2, BS = NCA * 32 * 2;   // bytes of one slice of a stage (K = 32)

// ---- digits of FP32 and FP64 values -------------------------------------------

template <typename T>
struct Dig;
template <>
struct Dig<double> {
  static constexpr int N = oz::kDigits, NBUF = 2;
  static constexpr uint32_t tmem = 512;
  static __device__ __forceinline__ void scan(double x, uint32_t& h, uint32_t& any) { oz::scan(oz::bits_of(x), h, any); }
  static __device__ __forceinline__ int code(uint32_t h, uint32_t any) { return oz::exp_code((int)(h >> 20), any != 0); }
  static __device__ __forceinline__ oz::Pair pair(double a, double b, int e) {
    return oz::Pair(oz::bits_of(a), oz::bits_of(b), e);
  }
  static __device__ __forceinline__ bool in_range(int ea, int eb) { return oz::in_range(ea, eb); }
};
// FP32: the cut to five digits (35 bits) and the dropped products (d > 4) err by
// at most 6 K 2^-35 u against K 2^-24 M of an FP32 sum: S_abs >= 48.
template <>
struct Dig<float> {
  static constexpr int N = 5, NBUF = 1;
  static constexpr uint32_t tmem = 256;
  static __device__ __forceinline__ void scan(float x, uint32_t& h, uint32_t& any) {
    const uint32_t b = __float_as_uint(x) & 0x7FFFFFFFu;
    h = max(h, b);
    any |= b;
  }
  static __device__ __forceinline__ int code(uint32_t h, uint32_t any) {
    const int e = (int)(h >> 23);
    return any == 0 ? oz::kZero : (e < 40 || e == 255) ? oz::kFar : e;
  }
  static __device__ __forceinline__ oz::Pair pair(float a, float b, int e) {
    // the same bits with the exponent where Pair looks for it
    const uint32_t ba = __float_as_uint(a), bb = __float_as_uint(b);
    auto wide = [](uint32_t x) {
      return ((unsigned long long)((x & 0x80000000u) | ((x >> 3) & 0x0FFFFFFFu)) << 32) | ((unsigned long long)(x & 7u) << 29);
    };
    return oz::Pair(wide(ba), wide(bb), e);
  }
  static __device__ __forceinline__ bool in_range(int ea, int eb) { return (unsigned)(ea + eb - 174) <= 190u; }
  static constexpr float abs_min = 64.f;
};

// All digit products of one stage into accumulators of NCA columns (S_abs behind them).
template <int N>
__device__ __forceinline__ void products(uint32_t tmem, uint32_t a, uint32_t b, bool first) {
  if constexpr (N == oz::kDigits) {
    oz::stage_mma<TR, NCA>(tmem, a, AS, b, first);
  } else {
#pragma unroll
    for (int kk = 0; kk < 2; ++kk) {
      const bool ow = first && kk == 0;
#pragma unroll
      for (int p = 0; p < N; ++p)
        oz::mma(tmem + NCA * p, oz::sdesc(a + p * AS + 256 * kk), oz::sdesc(b + 256 * kk), oz::idesc(TR, (N - p) * NCA),
                !(ow && p == 0));
      oz::mma(tmem + NCA * N, oz::sdesc(a + N * AS + 256 * kk), oz::sdesc(b + N * BS + 256 * kk), oz::idesc(TR, NCA), !ow);
    }
  }
}

// Four columns of the accumulators as values (0 where flagged), the flags as bits.
__device__ __forceinline__ uint32_t values4(uint32_t tacc, int ea, const int* eb, double (&v)[4]) {
  long long hi[4], lo[4];
  float sabs[4];
  oz::gather4<NCA>(tacc, hi, lo, sabs);
  uint32_t flag = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const bool fast = oz::in_range(ea, eb[i]) && sabs[i] >= oz::kAbsMin;
    v[i] = fast ? oz::assemble(hi[i], lo[i], ea + eb[i] - 2114) : 0.0;
    if (!fast && !oz::is_zero(ea, eb[i])) flag |= 1u << i;
  }
  return flag;
}
__device__ __forceinline__ uint32_t values4(uint32_t tacc, int ea, const int* eb, float (&v)[4]) {
  constexpr int N = Dig<float>::N;
  float w[N + 1][4];
#pragma unroll
  for (int d = 0; d <= N; ++d) oz::tmem_ld4(tacc + NCA * d, w[d]);
  oz::tmem_wait_ld();
  uint32_t flag = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float s = w[N - 1][i];
#pragma unroll
    for (int d = N - 2; d >= 0; --d) s = fmaf(s, 0.0078125f, w[d][i]);
    const bool fast = Dig<float>::in_range(ea, eb[i]) && w[N][i] >= Dig<float>::abs_min;
    v[i] = fast ? s * __uint_as_float((uint32_t)(ea + eb[i] - 266 + 127) << 23) : 0.f;
    if (!fast && !oz::is_zero(ea, eb[i])) flag |= 1u << i;
  }
  return flag;
}

// ---- leaves and merges ------------------------------------------------------------

template <typename T>
__global__ void __launch_bounds__(NT) leaf_copy_kernel(const Task* __restrict__ tasks, const Slot* __restrict__ slots) {
  const Task tk = tasks[blockIdx.x];
  const Node& nd = tk.nodes[tk.node];
  T* fb = (T*)slots[tk.slot].fbase;
  auto copy = [&](T* dst, const double* src, int64_t cnt) {
    for (int64_t e0 = threadIdx.x; e0 < cnt; e0 += 8 * NT) {
      double v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = e0 + q * NT < cnt ? __ldg(src + e0 + q * NT) : 0.0;
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (e0 + q * NT < cnt) dst[e0 + q * NT] = (T)v[q];
    }
  };
  if (!nd.leaf) return;
  const int part = blockIdx.y;   // D in four quarters of its columns, U, V
  if (part < 4) {
    const int64_t c0 = (int64_t)nd.n * part / 4, c1 = (int64_t)nd.n * (part + 1) / 4;
    copy(fb + nd.fD + c0 * nd.m, nd.D + c0 * nd.m, (c1 - c0) * nd.m);
  } else if (!nd.root) {
    if (part == 4) copy(fb + nd.fU, nd.U, (int64_t)nd.m * nd.ku);
    else copy(fb + nd.fV, nd.V, (int64_t)nd.n * nd.kv);
  }
}

// C (M x N, ld ldc) = A B in 32 x 32 tiles, K in chunks of 32: A(i, l) = a[i + l lda]
// (zero above the diagonal with tril), B(l, j) by the functor.
template <typename T, class LB>
__device__ void tile_mm(T* C, int ldc, const T* a, int lda, bool tril, LB lb, int M, int N, int K, T (*As)[33],
                        T (*Bs)[33]) {
  const int tid = threadIdx.x, r = tid & 31, q = tid >> 5;
  for (int i0 = 0; i0 < M; i0 += 32)
    for (int j0 = 0; j0 < N; j0 += 32) {
      T acc[4] = {T(0), T(0), T(0), T(0)};
      for (int k0 = 0; k0 < K; k0 += 32) {
        T va[4], vb[4];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const int e = tid + h * NT, i = e & 31, l = e >> 5;
          const bool oka = i0 + i < M && k0 + l < K && !(tril && k0 + l > i0 + i);
          va[h] = oka ? a[(i0 + i) + (int64_t)(k0 + l) * lda] : T(0);
          vb[h] = (k0 + i < K && j0 + l < N) ? lb(k0 + i, j0 + l) : T(0);
        }
        __syncthreads();
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const int e = tid + h * NT, i = e & 31, l = e >> 5;
          As[l][i] = va[h];
          Bs[l][i] = vb[h];   // Bs[j][k]
        }
        __syncthreads();
        const int kn = min(32, K - k0);
        for (int l = 0; l < kn; ++l) {
          const T x = As[l][r];
#pragma unroll
          for (int h = 0; h < 4; ++h) acc[h] = fma_t(x, Bs[q + 8 * h][l], acc[h]);
        }
      }
#pragma unroll
      for (int h = 0; h < 4; ++h)
        if (i0 + r < M && j0 + q + 8 * h < N) C[(i0 + r) + (int64_t)(j0 + q + 8 * h) * ldc] = acc[h];
    }
}

// The merge (src/ulvfactor.jl:74-79), one block per (node, product).  stage 0:
// T12 = U1 B12, T21 = U2 B21, U = [U1 R1; U2 R2], V = [V1 W1; V2 W2]; stage 1: the
// merged D = [D1, T12 V2^T; T21 V1^T, D2].
template <typename T>
__global__ void __launch_bounds__(NT) merge_kernel(const Task* __restrict__ tasks, const Slot* __restrict__ slots,
                                                   int stage) {
  __shared__ T As[32][33], Bs[32][33];
  const Task tk = tasks[blockIdx.x];
  const Node& nd = tk.nodes[tk.node];
  if (nd.leaf) return;
  T* fb = (T*)slots[tk.slot].fbase;
  const int part = blockIdx.y, h = part & 1;     // h: which child the product starts from
  const Node& c = tk.nodes[h ? nd.right : nd.left];
  const Node& o = tk.nodes[h ? nd.left : nd.right];
  const T* cU = fb + c.fU + c.mk;
  const T* cV = fb + c.fV + c.nk;
  const int m1 = tk.nodes[nd.left].mr, n1 = tk.nodes[nd.left].nr;   // offsets of the second child
  auto gen = [](const double* p, int ld) {
    return [p, ld](int l, int j) { return (T)__ldg(p + l + (int64_t)j * ld); };
  };
  if (stage == 0) {
    if (part < 2)
      tile_mm(fb + (h ? nd.fT21 : nd.fT12), c.mr, cU, c.m, c.lower_u != 0, gen(h ? nd.B21 : nd.B12, c.ku), c.mr, o.kv,
              c.ku, As, Bs);
    else if (nd.root)
      return;
    else if (part < 4)
      tile_mm(fb + nd.fU + (h ? m1 : 0), nd.m, cU, c.m, c.lower_u != 0, gen(h ? nd.R2 : nd.R1, c.ku), c.mr, nd.ku, c.ku,
              As, Bs);
    else
      tile_mm(fb + nd.fV + (h ? n1 : 0), nd.n, cV, c.n, false, gen(h ? nd.W2 : nd.W1, c.kv), c.nr, nd.kv, c.kv, As, Bs);
    return;
  }
  if (part < 2) {   // U_h B V_o^T: rows of child h, columns of the other
    const T* oV = fb + o.fV + o.nk;
    const int ldv = o.n;
    tile_mm(fb + nd.fD + (h ? m1 : 0) + (int64_t)(h ? 0 : n1) * nd.m, nd.m, fb + (h ? nd.fT21 : nd.fT12), c.mr, false,
            [oV, ldv](int l, int j) { return oV[j + (int64_t)l * ldv]; }, c.mr, o.nr, o.kv, As, Bs);
  } else {
    const T* src = fb + c.fD + c.mk + (int64_t)c.nk * c.m;
    T* dst = fb + nd.fD + (h ? m1 + (int64_t)n1 * nd.m : 0);
    for (int e = threadIdx.x; e < c.mr * c.nr; e += NT) {
      const int i = e % c.mr, j = e / c.mr;
      dst[i + (int64_t)j * nd.m] = src[i + (int64_t)j * c.m];
    }
  }
}

// ---- panels --------------------------------------------------------------------------

// Strictly upper Gram matrix of the reflectors in Yc (reflector-major, zero-padded
// to a multiple of 4), each of its 496 entries by one thread.
template <typename T, int NTH>
__device__ __forceinline__ void gram(const T* Yc, int YP, int len, T* G) {
  for (int e = threadIdx.x; e < 496; e += NTH) {
    // rows i and 30 - i of the strictly upper triangle make 32 entries
    const int i = e >> 5, j = e & 31;
    const int a = e >= 480 ? 15 : (j < 31 - i ? i : 30 - i), b = e >= 480 ? 16 + j : (j < 31 - i ? i + 1 + j : j);
    T s0 = T(0), s1 = T(0);
    for (int c = 0; c < len; c += 4) {
      T ya[4], yb[4];
      ld4(ya, Yc + a * YP + c);
      ld4(yb, Yc + b * YP + c);
      s0 = fma_t(ya[0], yb[0], s0);
      s1 = fma_t(ya[1], yb[1], s1);
      s0 = fma_t(ya[2], yb[2], s0);
      s1 = fma_t(ya[3], yb[3], s1);
    }
    G[a * GP + b] = s0 + s1;
  }
  __syncthreads();
}

template <typename T, int S>
constexpr size_t panel_smem() {
  return sizeof(T) * ((size_t)BP * (S + 4) + 2 * BP * GP);
}

// QL: columns c0 .. c0 + 31 of U (panel p from the last), reflector of column c
// with its pivot at row mk + c; LQ: rows i0 .. i0 + 31 of D[0:mk, :].  PL lanes per
// column (row), S / PL entries each in registers.  Reflectors are applied one at a
// time; each is published in shared memory with an mbarrier of its own, so that a
// warp waits for the next reflector only, not for the slower warps: the chain is
// the owner's apply and generate, and the other warps' FP64 instructions fill the
// pipes beside it.  FP64 with no more blocks than SMs takes 16 lanes per column
// (a shorter chain; no other block wants the pipes).
template <typename T, int S, bool QL, int PL>
__global__ void __launch_bounds__(32 * PL) panel_kernel(const Task* __restrict__ tasks, const Slot* __restrict__ slots, int p) {
  extern __shared__ __align__(16) unsigned char psm[];
  __shared__ __align__(8) uint64_t s_bar[BP];
  __shared__ T ptau[BP];
  constexpr int PE = S / PL, YP = S + 4;
  const Task tk = tasks[blockIdx.x];
  const Node& nd = tk.nodes[tk.node];
  if (nd.root || nd.mk == 0) return;
  const int m = nd.m, n = nd.n, k = nd.k, mk = nd.mk;
  const int e1 = QL ? k - BP * p : min(mk, BP * (p + 1)), e0 = QL ? max(0, e1 - BP) : BP * p, nb = e1 - e0;
  if (nb <= 0) return;
  const Slot& sl = slots[tk.slot];
  T* fb = (T*)sl.fbase;
  const int len = QL ? m : n;
  T* Yc = (T*)psm;   // the reflectors, explicitly: BP x S, ld YP
  T* G = Yc + BP * YP;
  T* Tm = G + BP * GP;
  const int tid = threadIdx.x, lane = tid & 31, g = tid / PL, l8 = tid % PL;
  const unsigned gm = (PL == 8 ? 0xFFu : 0xFFFFu) << (lane & (32 - PL));
  auto gsum = [&](T v) {
    if constexpr (PL == 16) v += __shfl_xor_sync(gm, v, 8);
    return gsum8(v, gm);
  };
  // entry t of this lane: row (column) l8 + PL t of column (row) e0 + g
  T* base = QL ? fb + nd.fU + (int64_t)(e0 + g) * m : fb + nd.fD + e0 + g;
  const int64_t step = QL ? 1 : m;
  T u[PE];
#pragma unroll
  for (int t = 0; t < PE; ++t) {
    const int i = l8 + PL * t;
    u[t] = (g < nb && i < len) ? base[i * step] : T(0);
  }
  if (tid < BP) oz::mbar_init(&s_bar[tid]);
  asm volatile("fence.mbarrier_init.release.cluster;");
  for (int e = tid; e < (BP - nb) * YP; e += 32 * PL) Yc[nb * YP + e] = T(0);
  __syncthreads();
  T* taus = fb + (QL ? nd.ftq : nd.ftl) + e0;
  // pivot of the panel's reflector a, and whether entry i belongs to its tail
  auto pivot = [&](int a) { return QL ? mk + e0 + a : e0 + a; };
  auto tail = [&](int i, int pv) { return QL ? i < pv : i > pv; };
  auto gen = [&](int a) {   // the PL lanes of column (row) a
    const int pv = pivot(a);
    T sq[2] = {T(0), T(0)}, mine = T(0);
#pragma unroll
    for (int t = 0; t < PE; ++t) {
      const int i = l8 + PL * t;
      if (tail(i, pv)) sq[t & 1] = fma_t(u[t], u[t], sq[t & 1]);
      if (i == pv) mine = u[t];
    }
    const T ss = gsum(sq[0] + sq[1]);
    const T alpha = __shfl_sync(gm, mine, (lane & (32 - PL)) | (pv & (PL - 1)));
    T beta, tau, sc;
    larfg_t(alpha, ss, beta, tau, sc);
#pragma unroll
    for (int t = 0; t < PE; ++t) {
      const int i = l8 + PL * t;
      const bool in = tail(i, pv);
      if (in) u[t] *= sc;   // 1 where tau is 0
      Yc[a * YP + i] = in ? u[t] : (i == pv ? T(1) : T(0));
      if (i == pv) u[t] = beta;
    }
    if (l8 == 0) {
      ptau[a] = tau;
      taus[a] = tau;
    }
    __syncwarp(gm);
    if (l8 == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(oz::smem_u32(&s_bar[a])) : "memory");
  };
  const int first = QL ? nb - 1 : 0;
  if (g == first) gen(first);
  __syncwarp();
  // the warp's columns (rows) are g0 .. g1; its last reflector to apply comes before its last column's own
  const int g0 = tid / 32 * (32 / PL), g1 = min(nb - 1, g0 + 32 / PL - 1);
  bool ok = true;
  for (int s = 0; s < nb; ++s) {
    const int a = QL ? nb - 1 - s : s, next = QL ? a - 1 : a + 1;
    if (QL ? a <= g0 : a >= g1) break;   // uniform over the warp
    ok = oz::mbar_wait(&s_bar[a], 0) && ok;
    __syncwarp();
    const T tau = ptau[a];
    const bool todo = QL ? g < a : (g > a && g < nb);
    if (todo) {   // tau = 0 leaves the column as it is
      T w0 = T(0), w1 = T(0);
      T vv[PE];
#pragma unroll
      for (int t = 0; t < PE; ++t) vv[t] = Yc[a * YP + l8 + PL * t];
#pragma unroll
      for (int t = 0; t < PE; t += 2) {
        w0 = fma_t(vv[t], u[t], w0);
        w1 = fma_t(vv[t + 1], u[t + 1], w1);
      }
      const T w = gsum(w0 + w1) * -tau;
#pragma unroll
      for (int t = 0; t < PE; ++t) u[t] = fma_t(w, vv[t], u[t]);
    }
    if (next >= 0 && next < nb && g == next) gen(next);
    __syncwarp();
  }
  if (!ok && sl.err) atomicCAS(sl.err, DEV_OK, DEV_TIMEOUT);
  // back to storage
#pragma unroll
  for (int t = 0; t < PE; ++t) {
    const int i = l8 + PL * t;
    if (g < nb && i < len) base[i * step] = u[t];
  }
  __syncthreads();
  if (!QL) {   // the reflectors as columns of Qt
    T* gQt = fb + nd.fQt + (int64_t)e0 * n;
    for (int e = tid; e < nb * n; e += 32 * PL) gQt[e] = Yc[e / n * YP + e % n];
  }
  gram<T, 32 * PL>(Yc, YP, len, G);
  T* Tg = fb + (QL ? nd.fTq : nd.fTl) + (int64_t)p * 1024;
  if constexpr (sizeof(T) == 8) blk_tmat_halves<32 * PL>(nb, G, ptau, Tm, Tg);
  else blk_tmat(nb, G, ptau, Tm, Tg);
}

// ---- block updates ----------------------------------------------------------------------

template <typename T>
struct ApplySmem {
  static constexpr int stage = (Dig<T>::N + 1) * (AS + BS);
  static constexpr int xs = TR * 33 * (int)sizeof(T);
  static constexpr int total = Dig<T>::NBUF == 2 ? 2 * stage : stage + xs;   // two stages: X overlays the first
  static_assert(xs <= (Dig<T>::N + 1) * AS, "X fits where a stage's A slices are");
};

// S <- S - ((S Y^T) T') Y for the panel's nb reflectors Y (nb x len), S in row
// tiles of 128: QL: the rows of S are the columns of D and the columns of U left
// of the panel, T' = T^T; LQ: the rows of D below the panel and the columns of V,
// T' = T.  Three products: X = S Y^T (K = len), Z = X T' (K = 32), Z Y (K = 32,
// columns in tiles of 32).  512 threads; a warp cuts 8 rows of S, 4 lanes per row
// with pairs of neighbouring entries, which reads 64 consecutive bytes in either
// orientation.  Cutting and putting together are bound by integer instructions
// (one FP64 product of 128 x 32: about 6 K clocks each for 128 rows), so warps
// whose rows lie beyond the tile's skip both.
template <typename T, bool QL>
__global__ void __launch_bounds__(AT, (sizeof(T) == 4 ? 2 : 1))
    apply_kernel(const Task* __restrict__ tasks, const Slot* __restrict__ slots, int p, int ntile) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ uint32_t s_tmem;
  __shared__ __align__(8) uint64_t s_done[2];
  __shared__ int s_row[TR], s_col[2][NCA];
  __shared__ int s_fail;
  using D = Dig<T>;
  constexpr int STAGE = ApplySmem<T>::stage, NBUF = D::NBUF, N = D::N;
  const Task tk = tasks[blockIdx.x / ntile];
  const Node& nd = tk.nodes[tk.node];
  if (nd.root || nd.mk == 0) return;
  const Slot& sl = slots[tk.slot];
  T* fb = (T*)sl.fbase;
  const int m = nd.m, n = nd.n, k = nd.k, mk = nd.mk, t0 = (blockIdx.x % ntile) * TR;
  const int e1 = QL ? k - BP * p : min(mk, BP * (p + 1)), e0 = QL ? max(0, e1 - BP) : BP * p, nb = e1 - e0;
  const int ra = QL ? n : m - e1;                    // rows from D, then from U or V
  const int rows = nb > 0 ? ra + (QL ? e0 : nd.kv) : 0;
  if (t0 >= rows) return;
  const int rt = min(TR, rows - t0);
  const int lb = QL ? 0 : e0, len = (QL ? min(m, mk + e1) : n) - lb;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  // S(i, l) = row_ptr(i)[l * row_step(i)]
  auto row_ptr = [&](int i) -> T* {
    if (QL) return i < ra ? fb + nd.fD + (int64_t)i * m : fb + nd.fU + (int64_t)(i - ra) * m;
    return (i < ra ? fb + nd.fD + e1 + i + (int64_t)lb * m : fb + nd.fV + (int64_t)(i - ra) * n + lb);
  };
  auto row_step = [&](int i) -> int64_t { return QL || i >= ra ? 1 : m; };
  const T* gU = fb + nd.fU + (int64_t)e0 * m;
  const T* gQt = fb + nd.fQt + (int64_t)e0 * n + lb;
  auto yval = [&](int a, int l) -> T {   // reflector a of the panel, entry lb + l
    if (a >= nb || l >= len) return T(0);
    if (!QL) return gQt[l + (int64_t)a * n];
    const int pv = mk + e0 + a;
    return l < pv ? gU[l + (int64_t)a * m] : (l == pv ? T(1) : T(0));
  };
  const T* gT = fb + (QL ? nd.fTq : nd.fTl) + (int64_t)p * 1024;
  auto tval = [&](int a, int b) -> T { return QL ? gT[a + b * BP] : gT[b + a * BP]; };   // T'(b, a)

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(oz::smem_u32(&s_tmem)),
                 "r"(D::tmem));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    oz::mbar_init(&s_done[0]);
    oz::mbar_init(&s_done[1]);
    asm volatile("fence.mbarrier_init.release.cluster;");
    s_fail = 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = s_tmem;

  uint32_t use = 0;   // stages issued; stage u uses buffer u % NBUF and barrier u & 1
  auto wait_use = [&](uint32_t u) {
    if (!oz::mbar_wait(&s_done[u & 1], (u >> 1) & 1)) s_fail = 1;
  };
  auto abuf = [&](uint32_t u) { return smem + (u % NBUF) * STAGE; };
  auto bbuf = [&](uint32_t u) { return smem + (u % NBUF) * STAGE + (N + 1) * AS; };
  auto issue = [&](const unsigned char* a, const unsigned char* b, bool first) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;");
      products<N>(tmem, oz::smem_u32(a), oz::smem_u32(b), first);
      oz::mma_commit(&s_done[use & 1]);
    }
    ++use;
  };
  auto put = [&](unsigned char* dst, int stride, const oz::Pair& pr) {
#pragma unroll
    for (int d = 0; d < N; ++d) *reinterpret_cast<uint32_t*>(dst + d * stride) = pr.digit(d);
    *reinterpret_cast<uint32_t*>(dst + N * stride) = pr.top_abs();
  };
  // cutting A: row 8 warp + lane / 4; cutting B: column tid / 16, pair tid % 16
  const int lr = 8 * warp + (lane >> 2), bc = tid >> 4, bj = tid & 15;
  const bool cutter = 8 * warp < rt;   // uniform over the warp
  auto row_code = [&](uint32_t h, uint32_t any) {
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      h = max(h, __shfl_xor_sync(0xffffffffu, h, o));
      any |= __shfl_xor_sync(0xffffffffu, any, o);
    }
    const int c = D::code(h, any);
    if ((lane & 3) == 0) s_row[lr] = c;
    return c;
  };
  auto col_code = [&](uint32_t h, uint32_t any, int buf) {
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
      h = max(h, __shfl_xor_sync(0xffffffffu, h, o));
      any |= __shfl_xor_sync(0xffffffffu, any, o);
    }
    const int c = D::code(h, any);
    if (bj == 0) s_col[buf][bc] = c;
    return c;
  };
  // results: row 32 (warp % 4) + lane, columns 8 (warp / 4) .. + 7
  const int orow = 32 * (warp & 3) + lane, oc0 = 8 * (warp >> 2);
  const uint32_t tacc = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)oc0;
  const bool oin = orow < rt, reader = 32 * (warp & 3) < rt;
  // the finished product's values of this thread; flagged ones by dot(row, column)
  auto collect = [&](T (&v)[8], int buf, auto dot) {
    wait_use(use - 1);
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (reader) {
      __syncwarp();
      const int ea = oin ? s_row[orow] : oz::kZero;
      uint32_t flag = 0;
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        T w[4];
        flag |= values4(tacc + 4 * g, ea, &s_col[buf][oc0 + 4 * g], w) << (4 * g);
#pragma unroll
        for (int i = 0; i < 4; ++i) v[4 * g + i] = w[i];
      }
      for (uint32_t rs = __ballot_sync(0xffffffffu, flag != 0); rs; rs &= rs - 1) {
        const int src = __ffs(rs) - 1;
#pragma unroll 1
        for (uint32_t cols = __shfl_sync(0xffffffffu, flag, src); cols; cols &= cols - 1) {
          const int i = __ffs(cols) - 1;
          T t = dot(32 * (warp & 3) + src, oc0 + i);
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (lane == src && j == i) v[j] = t;
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = T(0);
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
  };

  // ---- X = S Y^T ----
  T acc[8];
  {
    const int srow = t0 + lr;
    const bool sin = lr < rt;
    const T* sp = row_ptr(sin ? srow : t0);
    const int64_t ss = row_step(sin ? srow : t0);
    for (int c0 = 0; c0 < len; c0 += 128) {
      const int kc = min(128, len - c0), nst = (kc + 31) / 32;
      T v[16][2], y[4][2];
      uint32_t h = 0, any = 0, hy = 0, anyy = 0;
#pragma unroll
      for (int q = 0; q < 16; ++q)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int l = 8 * q + 2 * (lane & 3) + e;
          v[q][e] = sin && l < kc ? sp[(c0 + l) * ss] : T(0);
        }
#pragma unroll
      for (int s = 0; s < 4; ++s)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int l = 32 * s + 2 * bj + e;
          y[s][e] = l < kc ? yval(bc, c0 + l) : T(0);
        }
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        D::scan(v[q][0], h, any);
        D::scan(v[q][1], h, any);
      }
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        D::scan(y[s][0], hy, anyy);
        D::scan(y[s][1], hy, anyy);
      }
      const int ea = row_code(h, any), eb = col_code(hy, anyy, 0);
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        if (s < nst) {
          if (use >= NBUF) wait_use(use - NBUF);
          unsigned char* a = abuf(use);
          unsigned char* b = bbuf(use);
          if (cutter) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
              put(a + oz::core_off(lr, q) + 4 * (lane & 3), AS, D::pair(v[4 * s + q][0], v[4 * s + q][1], ea));
          }
          put(b + oz::core_off(bc, bj >> 2) + 4 * (bj & 3), BS, D::pair(y[s][0], y[s][1], eb));
          issue(a, b, s == 0);
        }
      }
      T d[8];
      collect(d, 0, [&](int i, int a) {
        const T* q = row_ptr(t0 + i) + c0 * row_step(t0 + i);
        T t = T(0);
        for (int l = lane; l < kc; l += 32) t = fma_t(q[l * row_step(t0 + i)], yval(a, c0 + l), t);
        return t;
      });
      if (c0 == 0) {
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] = d[i];
      } else {
        asm volatile("");
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] += d[i];
      }
      __syncthreads();   // the accumulators and the codes may be overwritten
      asm volatile("tcgen05.fence::after_thread_sync;");
    }
  }
  // every MMA so far is done: buffers are free; with two, X takes the first's place
  T* Xs = (T*)(NBUF == 2 ? smem : smem + STAGE);
#pragma unroll
  for (int i = 0; i < 8; ++i) Xs[orow * 33 + oc0 + i] = oin ? acc[i] : T(0);
  __syncthreads();
  unsigned char* A1 = smem + (NBUF - 1) * STAGE;
  auto cut_x = [&]() {
    T v[4][2];
    uint32_t h = 0, any = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        v[q][e] = Xs[lr * 33 + 8 * q + 2 * (lane & 3) + e];
        D::scan(v[q][e], h, any);
      }
    const int ea = row_code(h, any);
    if (cutter) {
#pragma unroll
      for (int q = 0; q < 4; ++q) put(A1 + oz::core_off(lr, q) + 4 * (lane & 3), AS, D::pair(v[q][0], v[q][1], ea));
    }
  };
  auto cut_b = [&](T x0, T x1, int buf, unsigned char* b) {   // column bc, K pair bj
    uint32_t h = 0, any = 0;
    D::scan(x0, h, any);
    D::scan(x1, h, any);
    const int eb = col_code(h, any, buf);
    put(b + oz::core_off(bc, bj >> 2) + 4 * (bj & 3), BS, D::pair(x0, x1, eb));
  };
  unsigned char* B1 = A1 + (N + 1) * AS;
  // ---- Z = X T' ----
  cut_x();
  cut_b(tval(bc, 2 * bj), tval(bc, 2 * bj + 1), 0, B1);
  issue(A1, B1, true);
  T z[8];
  collect(z, 0, [&](int i, int a) { return Xs[i * 33 + lane] * tval(a, lane); });
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; ++i) Xs[orow * 33 + oc0 + i] = oin ? z[i] : T(0);
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  // ---- S -= Z Y, 32 columns at a time ----
  cut_x();
  {
    T* sp = row_ptr(t0 + (oin ? orow : 0));
    const int64_t ss = row_step(t0 + (oin ? orow : 0));
    unsigned char* B0 = smem + (N + 1) * AS;   // with two buffers the tiles of Y alternate between them
    T y0 = yval(2 * bj, bc), y1 = yval(2 * bj + 1, bc);
    for (int l0 = 0, j = 0; l0 < len; l0 += 32, ++j) {
      unsigned char* b = NBUF == 2 && (j & 1) ? B0 : B1;
      cut_b(y0, y1, j & 1, b);
      issue(A1, b, true);
      // the next tile of Y and this tile of S while the products run
      y0 = yval(2 * bj, l0 + 32 + bc);
      y1 = yval(2 * bj + 1, l0 + 32 + bc);
      T old[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) old[i] = oin && l0 + oc0 + i < len ? sp[(l0 + oc0 + i) * ss] : T(0);
      T d[8];
      collect(d, j & 1, [&](int i, int c) { return Xs[i * 33 + lane] * yval(lane, l0 + c); });
      if (reader) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (oin && l0 + oc0 + i < len) sp[(l0 + oc0 + i) * ss] = old[i] - d[i];
      }
      __syncthreads();   // the accumulators may be overwritten
      asm volatile("tcgen05.fence::after_thread_sync;");
    }
  }
  if (s_fail && tid == 0 && sl.err) atomicCAS(sl.err, DEV_OK, DEV_TIMEOUT);
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(D::tmem));
}

// ---- roots ------------------------------------------------------------------------------

// The roots' LU with partial pivoting, in shared memory where it fits.
template <typename T>
__global__ void __launch_bounds__(NT) root_kernel(const Task* __restrict__ tasks, const Slot* __restrict__ slots,
                                                  int smem_rows) {
  extern __shared__ __align__(16) unsigned char fsm[];
  __shared__ T s_l[2 * 512];
  __shared__ int s_piv[2];
  const Task tk = tasks[blockIdx.x];
  const Node& nd = tk.nodes[tk.node];
  if (!nd.root) return;
  const Slot& sl = slots[tk.slot];
  T* fb = (T*)sl.fbase;
  T* gD = fb + nd.fD;
  const int m = nd.m, tid = threadIdx.x;
  int32_t* piv = (int32_t*)(fb + nd.fpiv);
  if (m > smem_rows) {
    lu_blk(gD, m, m, piv, sl.err, s_l, s_piv);
    return;
  }
  T* sD = (T*)fsm;
  const int ld = m | 1;
  for (int e = tid; e < m * m; e += NT) sD[(e % m) + (e / m) * ld] = gD[e];
  __syncthreads();
  lu_blk(sD, m, ld, piv, sl.err, s_l, s_piv);
  for (int e = tid; e < m * m; e += NT) gD[e] = sD[(e % m) + (e / m) * ld];
}

template <typename T, int S, bool QL, int PL>
cudaError_t panel_sized(const Task* t, int64_t nt, const Slot* s, int p, cudaStream_t st) {
  constexpr size_t smem = panel_smem<T, S>();
  auto* k = panel_kernel<T, S, QL, PL>;
  static SmemOptIn opt_in;
  const cudaError_t e = opt_in((const void*)k, smem);
  if (e != cudaSuccess) return e;
  k<<<(unsigned)nt, 32 * PL, smem, st>>>(t, s, p);
  return cudaGetLastError();
}
template <typename T, bool QL>
cudaError_t panel(const Task* t, int64_t nt, const Slot* s, int p, int len, int sms, cudaStream_t st) {
  if constexpr (sizeof(T) == 8) {
    if (nt <= sms && len <= 64) return panel_sized<T, 64, QL, 16>(t, nt, s, p, st);
    if (nt <= sms && len <= 128) return panel_sized<T, 128, QL, 16>(t, nt, s, p, st);
    if (nt <= sms && len <= 256) return panel_sized<T, 256, QL, 16>(t, nt, s, p, st);
  }
  if (len <= 64) return panel_sized<T, 64, QL, 8>(t, nt, s, p, st);
  if (len <= 128) return panel_sized<T, 128, QL, 8>(t, nt, s, p, st);
  if (len <= 256) return panel_sized<T, 256, QL, 8>(t, nt, s, p, st);
  return panel_sized<T, 512, QL, 8>(t, nt, s, p, st);
}
template <typename T, bool QL>
cudaError_t apply(const Task* t, int64_t nt, const Slot* s, int p, int rows, cudaStream_t st) {
  if (rows <= 0) return cudaSuccess;
  static SmemOptIn opt_in;
  const cudaError_t e = opt_in((const void*)apply_kernel<T, QL>, ApplySmem<T>::total);
  if (e != cudaSuccess) return e;
  const int ntile = (rows + TR - 1) / TR;
  apply_kernel<T, QL><<<(unsigned)(nt * ntile), AT, ApplySmem<T>::total, st>>>(t, s, p, ntile);
  return cudaGetLastError();
}

}  // namespace

bool factor_pan_fits(int mmax, int nmax) { return mmax <= 512 && nmax <= 512; }

template <typename T>
cudaError_t launch_ulv_factor_pan(const Task* t, int64_t nt, const Slot* s, const FactorDims& d, int sms, int* launches,
                                  cudaStream_t st) {
  *launches = 0;
  if (nt <= 0) return cudaSuccess;
  cudaError_t e = cudaSuccess;
  // the launches in order, none after one that failed
  auto step = [&](auto launch) {
    if (e == cudaSuccess) e = launch_fault();
    if (e == cudaSuccess) e = launch();
    ++*launches;
  };
  if (d.leaves)
    step([&] {
      leaf_copy_kernel<T><<<dim3((unsigned)nt, 6), NT, 0, st>>>(t, s);
      return cudaGetLastError();
    });
  for (int stage = 0; d.branches && stage < 2; ++stage)
    step([&] {
      merge_kernel<T><<<dim3((unsigned)nt, stage == 0 ? 6 : 4), NT, 0, st>>>(t, s, stage);
      return cudaGetLastError();
    });
  for (int p = 0; p * BP < d.kmax; ++p) {
    step([&] { return panel<T, true>(t, nt, s, p, d.mmax, sms, st); });
    step([&] { return apply<T, true>(t, nt, s, p, d.nmax + std::max(0, d.kmax - BP * (p + 1)), st); });
  }
  for (int p = 0; p * BP < d.mkmax; ++p) {
    step([&] { return panel<T, false>(t, nt, s, p, d.nmax, sms, st); });
    step([&] { return apply<T, false>(t, nt, s, p, d.mmax + d.kvmax, st); });
  }
  if (d.rootmax > 0) {
    const int cap = (int)(200 * 1024 / sizeof(T));
    const int rows = d.rootmax * (d.rootmax | 1) <= cap ? d.rootmax : 0;
    step([&] {
      static SmemOptIn opt_in;
      const cudaError_t r = opt_in((const void*)root_kernel<T>, cap * sizeof(T));
      if (r != cudaSuccess) return r;
      root_kernel<T><<<(unsigned)nt, NT, (size_t)rows * (rows | 1) * sizeof(T), st>>>(t, s, rows);
      return cudaGetLastError();
    });
  }
  return e;
}

template cudaError_t launch_ulv_factor_pan<double>(const Task*, int64_t, const Slot*, const FactorDims&, int, int*,
                                                   cudaStream_t);
template cudaError_t launch_ulv_factor_pan<float>(const Task*, int64_t, const Slot*, const FactorDims&, int, int*,
                                                  cudaStream_t);

}  // namespace hss
