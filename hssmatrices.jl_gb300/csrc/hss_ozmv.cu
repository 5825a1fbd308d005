// HSS x dense product (reference src/matmul.jl:13-62) in FP64 accuracy on the
// tensor cores (hss_oz.cuh), one launch per tree level.
//
// Every step of the product multiplies a node's generators, stacked, with a
// tall block of columns:
//   OZ_UP_LEAF    [D; V^T] X                      C = alpha D X + beta Y, Z = V^T X  (:34, :46)
//   OZ_UP_BRANCH  [[W1^T W2^T]; [0 B12]; [B21 0]] [Z1; Z2]
//                                                 Z_p, and G1, G2 into the children's F  (:39, :51, :55)
//   OZ_DOWN       [R1; R2] F_p                    F_c += R_c F_p  (:50-56)
//   OZ_FINAL      U F                             C += alpha U F, column sums of squares  (:47)
// The digit slices of the stacked generators are made once per plan
// (ozmv_prep_kernel), in the operand layout, 20 bytes per entry: per node and
// sweep, by tiles of 128 rows, chunks of K <= 128 and stages of K = 32, with the
// row exponents of each chunk behind it.
//
// ozmv_kernel walks units (node, row tile, column tile of NC) with warps that
// have one job each and meet on mbarriers, so that the copies, the cutting of X,
// the MMAs and the outputs of neighbouring units overlap:
//   warp 0        bulk copies of A's slices into a ring of two stages;
//   warp 1        the digit products (oz::stage_mma), accumulators in tensor memory;
//   warps 2-5     X, 128 x NC per chunk, cut into digits next to A's;
//   warps 6-21    accumulators put together (and added up over chunks) in FP64,
//                 the check's FP64 sums, outputs.
// The 200 KB ring leaves one block per SM.  A launch after the first of a product
// starts while the one before it ends (programmatic dependent launch): its set-up
// and its first copies of A's slices, which no launch writes, come before the
// wait for the previous step's outputs; every block waits for that step before it
// ends, so that the chain of launches stays whole where a level has no units.  Waits
// are bounded: one that runs out records DEV_TIMEOUT and the block ends once
// its copies and MMAs have.
//
// Measured (one GB300, n = 65536, leaves of 128, k = 32): 32 columns 938 -> 287 us
// (the FP64 pipe needs 840 us), 64 columns 1838 -> 422; the residual of a refined
// solve at 32 columns 374 -> 290 us.  The slices are 330 MB, 49 us at the measured
// copy rate; beyond that the time is latency: leaves 88 us and 43 us for the two
// passes, about 8 us for each of the 17 steps between them (start of the grid,
// descriptors, X, the digits' MMAs, the outputs).  Sixteen output warps instead
// of eight, and no FP64 instruction that an output does not need, took the 32
// columns from 360 to 287 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "hss_internal.h"
#include "hss_launch.h"
#include "hss_optin.h"
#include "hss_oz.cuh"

namespace hss {

namespace {

constexpr int XW = 4;                  // warps that cut X
constexpr int EW = 16;                 // output warps
constexpr int OT = 32 * (2 + XW + EW); // threads
constexpr int TR = 128;                // rows per tile
constexpr int KC = 128;                // K per chunk
constexpr int KS = 32;                 // K per stage
constexpr int kASlice = TR * KS * 2;   // shared-memory bytes of one slice of a stage of A

template <int NC>
struct Ring {
  static constexpr int xslice = NC * KS * 2;
  static constexpr int stage = oz::kSlices * (kASlice + xslice);
  static constexpr int smem = 2 * stage;
  static constexpr uint32_t tmem = NC == 32 ? 512 : 256;   // (kAcc + 1) NC columns, a power of two
};

__host__ __device__ __forceinline__ int oz_rows(const Node& nd, int kind) {
  switch (kind) {
    case OZ_UP_LEAF: return nd.gm + nd.kv;
    case OZ_UP_BRANCH: return nd.kv + nd.cku[0] + nd.cku[1];
    case OZ_DOWN: return nd.cku[0] + nd.cku[1];
    default: return nd.gm;
  }
}
__host__ __device__ __forceinline__ int oz_inner(const Node& nd, int kind) {
  switch (kind) {
    case OZ_UP_LEAF: return nd.gn;
    case OZ_UP_BRANCH: return nd.ckv[0] + nd.ckv[1];
    default: return nd.ku;
  }
}
__host__ __device__ __forceinline__ int round8(int x) { return (x + 7) & ~7; }
// Bytes of chunk c of a tile of `rows` rows, K inner terms in all: slices, then row codes.
__host__ __device__ __forceinline__ int64_t oz_chunk_bytes(int rows, int K, int c) {
  const int kc = K - c * KC < KC ? K - c * KC : KC;
  return (int64_t)((kc + KS - 1) / KS) * oz::kSlices * round8(rows) * 64 + round8(rows) * 4;
}
__host__ __device__ __forceinline__ int64_t oz_tile_bytes(int rows, int K) {
  const int full = K / KC;
  int64_t b = full * oz_chunk_bytes(rows, KC, 0);
  if (K % KC) b += oz_chunk_bytes(rows, K, full);
  return b;
}

// Entry (row, k) of the stacked generators.
__device__ __forceinline__ double oz_entry(const Node& nd, int kind, int row, int k) {
  const double* p = nullptr;
  switch (kind) {
    case OZ_UP_LEAF: p = row < nd.gm ? nd.D + row + (int64_t)k * nd.gm : nd.V + k + (int64_t)(row - nd.gm) * nd.gn; break;
    case OZ_UP_BRANCH: {
      const int v1 = nd.ckv[0], i = row - nd.kv;
      if (i < 0) p = k < v1 ? nd.W1 + k + (int64_t)row * v1 : nd.W2 + (k - v1) + (int64_t)row * nd.ckv[1];
      else if (i < nd.cku[0]) p = k < v1 ? nullptr : nd.B12 + i + (int64_t)(k - v1) * nd.cku[0];
      else p = k < v1 ? nd.B21 + (i - nd.cku[0]) + (int64_t)k * nd.cku[1] : nullptr;
      break;
    }
    case OZ_DOWN:
      p = row < nd.cku[0] ? nd.R1 + row + (int64_t)k * nd.cku[0] : nd.R2 + (row - nd.cku[0]) + (int64_t)k * nd.cku[1];
      break;
    default: p = nd.U + row + (int64_t)k * nd.gm;
  }
  return p ? __ldg(p) : 0.0;
}

// One block per (task, row tile, chunk): the tile of stacked generators staged in
// shared memory (consecutive threads read consecutive entries of each block),
// then its slices and row codes.
constexpr int PT = 512;
constexpr int PLD = KC + 1;
constexpr int kPrepSmem = TR * PLD * 8;

__global__ void __launch_bounds__(PT) ozmv_prep_kernel(const Task* __restrict__ tasks, int kind, int ntile, int nchunk,
                                                       unsigned char* __restrict__ base) {
  extern __shared__ __align__(16) double tile[];   // tile[r PLD + k]
  __shared__ uint32_t s_h[PT / TR][TR], s_any[PT / TR][TR];
  const int c = blockIdx.x % nchunk, t0 = blockIdx.x / nchunk % ntile * TR;
  const Task tk = tasks[blockIdx.x / (nchunk * ntile)];
  const Node& nd = tk.nodes[tk.node];
  const int64_t off = kind <= OZ_UP_BRANCH ? nd.fozu : nd.fozd;
  const int rows = oz_rows(nd, kind), K = oz_inner(nd, kind), tid = threadIdx.x;
  const int rt = min(TR, rows - t0), kc = min(KC, K - c * KC);
  if (off < 0 || rt <= 0 || kc <= 0) return;
  const int r8 = round8(rt), nst = (kc + KS - 1) / KS;
  unsigned char* img = base + off + (int64_t)(t0 / TR) * oz_tile_bytes(TR, K);
  for (int i = 0; i < c; ++i) img += oz_chunk_bytes(rt, K, i);
  // rows of transposed blocks (V^T, W^T) are contiguous along k, the others' columns along the rows
  const int cut = kind == OZ_UP_LEAF ? nd.gm : kind == OZ_UP_BRANCH ? nd.kv : 0;
  const int mid = min(rt, max(0, cut - t0));
  auto stage = [&](int ra, int n, bool kfast) {
#pragma unroll 8
    for (int e = tid; e < n * kc; e += PT) {
      const int r = ra + (kfast ? e / kc : e % n), k = kfast ? e % kc : e / n;
      tile[r * PLD + k] = oz_entry(nd, kind, t0 + r, c * KC + k);
    }
  };
  if (mid > 0) stage(0, mid, kind == OZ_UP_BRANCH);
  if (mid < rt) stage(mid, rt - mid, kind == OZ_UP_LEAF);
  __syncthreads();
  const int r = tid & (TR - 1), q = tid / TR;
  uint32_t hmax = 0, any = 0;
  if (r < rt)
    for (int k = q; k < kc; k += PT / TR) oz::scan(oz::bits_of(tile[r * PLD + k]), hmax, any);
  s_h[q][r] = hmax;
  s_any[q][r] = any;
  __syncthreads();
  if (r >= r8) return;
#pragma unroll
  for (int i = 0; i < PT / TR; ++i) {
    hmax = max(hmax, s_h[i][r]);
    any |= s_any[i][r];
  }
  const int emax = (int)(hmax >> 20);
  if (q == 0) reinterpret_cast<int*>(img + (int64_t)nst * oz::kSlices * r8 * 64)[r] = oz::exp_code(emax, any != 0);
  for (int kg = q; kg < 4 * nst; kg += PT / TR) {
    uint4 w[oz::kSlices];
    uint32_t* ww = reinterpret_cast<uint32_t*>(w);
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      unsigned long long b[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int k = 8 * kg + 2 * h + e;
        b[e] = r < rt && k < kc ? oz::bits_of(tile[r * PLD + k]) : 0ull;
      }
      const oz::Pair pr(b[0], b[1], emax);
#pragma unroll
      for (int p = 0; p < oz::kDigits; ++p) ww[4 * p + h] = pr.digit(p);
      ww[4 * oz::kDigits + h] = pr.top_abs();
    }
    unsigned char* dst = img + (int64_t)(kg >> 2) * oz::kSlices * r8 * 64 + oz::core_off(r, kg & 3);
#pragma unroll
    for (int p = 0; p < oz::kSlices; ++p) *reinterpret_cast<uint4*>(dst + (int64_t)p * r8 * 64) = w[p];
  }
}

struct Unit {
  const Node* nd;
  const Slot* sl;
  int j0, nc;        // columns
  int t0, rt, K;     // rows of the tile, inner terms
  const unsigned char* img;
};

// Unit u of the launch; false when it is empty (a smaller node or slot of the level).
__device__ __forceinline__ bool unit_of(int64_t u, const Task* tasks, const Slot* slots, int kind, int ntile, int nchunk,
                                        int ncols, Unit& x) {
  const int ch = (int)(u % nchunk), t = (int)((u / nchunk) % ntile);
  const Task tk = tasks[u / ((int64_t)nchunk * ntile)];
  x.nd = &tk.nodes[tk.node];
  x.sl = &slots[tk.slot];
  x.j0 = ch * ncols;
  x.nc = min(ncols, x.sl->r - x.j0);
  if (x.nc <= 0) return false;
  const Node& nd = *x.nd;
  if (kind == OZ_UP_BRANCH && nd.leaf) return false;   // single-leaf trees among the roots
  if (kind == OZ_FINAL && nd.root) return false;
  const int rows = oz_rows(nd, kind);
  x.K = oz_inner(nd, kind);
  x.t0 = t * TR;
  x.rt = min(TR, rows - x.t0);
  if (x.rt <= 0 || (x.K == 0 && kind == OZ_DOWN)) return false;
  x.img = x.sl->oz + (kind <= OZ_UP_BRANCH ? nd.fozu : nd.fozd) + (int64_t)t * oz_tile_bytes(TR, x.K);
  return true;
}

// Bounded wait; the first poll does not block, so that a limit of one poll can
// run out.
__device__ __forceinline__ bool wait_bar(uint64_t* bar, uint32_t parity, uint32_t limit, volatile int* fail) {
  uint32_t done;
  asm volatile(
      "{\n.reg .pred q;\nmbarrier.test_wait.parity.shared::cta.b64 q, [%1], %2;\nselp.u32 %0, 1, 0, q;\n}\n"
      : "=r"(done)
      : "r"(oz::smem_u32(bar)), "r"(parity)
      : "memory");
  for (uint32_t it = 1; !done && it < limit && !*fail; ++it)
    asm volatile(
        "{\n.reg .pred q;\nmbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\nselp.u32 %0, 1, 0, q;\n}\n"
        : "=r"(done)
        : "r"(oz::smem_u32(bar)), "r"(parity)
        : "memory");
  if (!done) *fail = 1;
  return done != 0;
}
__device__ __forceinline__ void arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(oz::smem_u32(bar)) : "memory");
}

template <int NC>
__global__ void __launch_bounds__(OT, 1) ozmv_kernel(const Task* __restrict__ tasks, int64_t nunits, int ntile,
                                                     int nchunk, const Slot* __restrict__ slots, int kind,
                                                     uint32_t limit) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ uint32_t s_tmem;
  // the ring's stages: A in, X in, free; the accumulators: complete, read
  __shared__ __align__(8) uint64_t s_fa[2], s_fx[2], s_free[2], s_acc, s_read, s_drain;
  __shared__ int s_col[4][NC];
  __shared__ volatile int s_fail;
  using R = Ring<NC>;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(oz::smem_u32(&s_tmem)),
                 "r"(R::tmem));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 32) {
    for (int i = 0; i < 2; ++i) {
      oz::mbar_init(&s_fa[i]);
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(oz::smem_u32(&s_fx[i])), "r"(XW));
      oz::mbar_init(&s_free[i]);
    }
    oz::mbar_init(&s_acc);
    oz::mbar_init(&s_drain);
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(oz::smem_u32(&s_read)), "r"(EW));
    asm volatile("fence.mbarrier_init.release.cluster;");
    s_fail = 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = s_tmem;
  uint32_t use = 0;   // stages passed: ring half use & 1, its (use / 2)-th use
  asm volatile("griddepcontrol.launch_dependents;");

  if (warp == 0) {
    if (lane == 0) {
      for (int64_t u = blockIdx.x; u < nunits && !s_fail; u += gridDim.x) {
        Unit x;
        if (!unit_of(u, tasks, slots, kind, ntile, nchunk, NC, x)) continue;
        const uint32_t slice = round8(x.rt) * 64;
        const unsigned char* img = x.img;
        for (int c = 0; c * KC < x.K && !s_fail; ++c) {
          const int nst = (min(KC, x.K - c * KC) + KS - 1) / KS;
          for (int s = 0; s < nst && !s_fail; ++s, ++use) {
            const int h = use & 1;
            if (use >= 2 && !wait_bar(&s_free[h], ((use >> 1) - 1) & 1, limit, &s_fail)) break;
            unsigned char* dst = smem + h * R::stage;
            const unsigned char* src = img + (int64_t)s * oz::kSlices * slice;
            if (slice == kASlice) {
              oz::bulk_load(dst, src, oz::kSlices * kASlice, &s_fa[h]);
            } else {
              asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(oz::smem_u32(&s_fa[h])),
                           "r"(oz::kSlices * slice)
                           : "memory");
              for (int p = 0; p < oz::kSlices; ++p)
                asm volatile(
                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                        oz::smem_u32(dst + p * kASlice)),
                    "l"(src + p * slice), "r"(slice), "r"(oz::smem_u32(&s_fa[h]))
                    : "memory");
            }
          }
          img += oz_chunk_bytes(x.rt, x.K, c);
        }
      }
      if (s_fail)   // no copy may be in flight when the block ends
        for (uint32_t i = use > 2 ? use - 2 : 0; i < use; ++i) oz::mbar_wait(&s_fa[i & 1], (i >> 1) & 1);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      uint32_t chunk = 0;
      for (int64_t u = blockIdx.x; u < nunits && !s_fail; u += gridDim.x) {
        Unit x;
        if (!unit_of(u, tasks, slots, kind, ntile, nchunk, NC, x)) continue;
        for (int c = 0; c * KC < x.K && !s_fail; ++c, ++chunk) {
          const int nst = (min(KC, x.K - c * KC) + KS - 1) / KS;
          if (chunk >= 1 && !wait_bar(&s_read, (chunk - 1) & 1, limit, &s_fail)) break;
          for (int s = 0; s < nst; ++s, ++use) {
            const int h = use & 1;
            if (!wait_bar(&s_fa[h], (use >> 1) & 1, limit, &s_fail) ||
                !wait_bar(&s_fx[h], (use >> 1) & 1, limit, &s_fail))
              break;
            asm volatile("tcgen05.fence::after_thread_sync;");
            const uint32_t a = oz::smem_u32(smem + h * R::stage);
            oz::stage_mma<TR, NC>(tmem, a, kASlice, a + oz::kSlices * kASlice, s == 0);
            oz::mma_commit(&s_free[h]);
          }
          oz::mma_commit(&s_acc);
        }
      }
      if (s_fail) {
        oz::mma_commit(&s_drain);
        oz::mbar_wait(&s_drain, 0);
      }
    }
  } else if (warp < 2 + XW) {
    // X: thread (column col, K pairs 2 kq of K groups hs, hs + NH, ...)
    constexpr int NH = 8 * XW / NC;            // 4 NH threads per column, taking its K groups in turn
    constexpr int NP = 16 / NH;                // pairs per thread and chunk
    static_assert(NH <= 4, "every thread has a pair in every stage");
    const int t = tid - 64, col = t / (4 * NH), kq = t & 3, hs = (t >> 2) % NH;
    uint32_t chunk = 0;
    bool ok = true, waited = false;   // uniform over the warp, as is every wait's outcome
    for (int64_t u = blockIdx.x; u < nunits && ok; u += gridDim.x) {
      Unit x;
      if (!unit_of(u, tasks, slots, kind, ntile, nchunk, NC, x)) continue;
      const Node& nd = *x.nd;
      const Slot& sl = *x.sl;
      // X(k) = base[k] for k < split, base2[k] beyond
      const double *xb, *xb2;
      int64_t ldx;
      int split = x.K;
      if (kind == OZ_UP_LEAF) {
        ldx = sl.ldb;
        xb = sl.B + nd.col0;
        xb2 = xb;
      } else {
        ldx = sl.ldws;
        const double* ws = (const double*)sl.ws;
        if (kind == OZ_UP_BRANCH) {
          xb = ws + nd.cwz[0];
          split = nd.ckv[0];
          xb2 = ws + nd.cwz[1] - split;
        } else {
          xb = ws + nd.wf;
          xb2 = xb;
        }
      }
      const int64_t cofs = (int64_t)(x.j0 + col) * ldx;
      const bool cin = col < x.nc;
      if (!waited) {
        asm volatile("griddepcontrol.wait;" ::: "memory");   // the previous step's outputs
        waited = true;
      }
      for (int c = 0; c * KC < x.K && ok; ++c, ++chunk) {
        const int kc = min(KC, x.K - c * KC), nst = (kc + KS - 1) / KS;
        double v[2 * NP];
        uint32_t hmax = 0, any = 0;
#pragma unroll
        for (int i = 0; i < 2 * NP; ++i) {
          const int kg = hs + NH * (i >> 1), k = 8 * kg + 2 * kq + (i & 1), kk = c * KC + k;
          v[i] = cin && k < kc ? *((kk < split ? xb : xb2) + kk + cofs) : 0.0;
        }
#pragma unroll
        for (int i = 0; i < 2 * NP; ++i) oz::scan(oz::bits_of(v[i]), hmax, any);
        int emax = (int)(hmax >> 20);
#pragma unroll
        for (int o = 1; o < 4 * NH; o <<= 1) {
          emax = max(emax, __shfl_xor_sync(0xffffffffu, emax, o));
          any |= __shfl_xor_sync(0xffffffffu, any, o);
        }
        if (kq == 0 && hs == 0) s_col[chunk & 3][col] = oz::exp_code(emax, any != 0);
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          if (s < nst && ok) {
            const int h = use & 1;
            if (use >= 2) ok = __all_sync(0xffffffffu, wait_bar(&s_free[h], ((use >> 1) - 1) & 1, limit, &s_fail));
            if (!ok) continue;
            unsigned char* dst = smem + h * R::stage + oz::kSlices * kASlice;
#pragma unroll
            for (int i = 0; i < NP / 4; ++i) {
              const int q = s * (NP / 4) + i, kg = (hs + NH * q) & 3;
              const oz::Pair pr(oz::bits_of(v[2 * q]), oz::bits_of(v[2 * q + 1]), emax);
              unsigned char* d = dst + oz::core_off(col, kg) + 4 * kq;
#pragma unroll
              for (int p = 0; p < oz::kDigits; ++p) *reinterpret_cast<uint32_t*>(d + p * R::xslice) = pr.digit(p);
              *reinterpret_cast<uint32_t*>(d + oz::kDigits * R::xslice) = pr.top_abs();
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) arrive(&s_fx[h]);
            ++use;
          }
        }
      }
    }
  } else {
    // outputs: row 32 (warp % 4) + lane of the tile, CW columns
    constexpr int CW = 4 * NC / EW;
    const int lrow = 32 * (warp & 3) + lane, cw0 = CW * ((warp - 2 - XW) >> 2);
    const uint32_t tacc = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)cw0;
    uint32_t chunk = 0;
    bool ok = true, waited = false;
    for (int64_t u = blockIdx.x; u < nunits && ok; u += gridDim.x) {
      Unit x;
      if (!unit_of(u, tasks, slots, kind, ntile, nchunk, NC, x)) continue;
      const Node& nd = *x.nd;
      const Slot& sl = *x.sl;
      const bool rin = lrow < x.rt;
      const int nc = min(CW, x.nc - cw0);   // this warp's columns (may be <= 0)
      // where this row goes: the workspace, or C; and the term it is added to
      const int row = x.t0 + lrow;
      const bool toc = kind == OZ_FINAL || (kind == OZ_UP_LEAF && row < nd.gm);
      const int64_t j0 = x.j0 + cw0;
      double* out;
      const double* old;
      int64_t ldo, ldy;
      double alpha = 1.0, beta = 0.0;
      if (toc) {
        out = sl.C + nd.row0 + row + j0 * sl.ldc;
        ldo = sl.ldc;
        alpha = sl.alpha;
        // beta Y, or the leaf product that the first launch wrote
        beta = kind == OZ_FINAL ? 1.0 : sl.beta;
        old = kind == OZ_FINAL ? out : sl.Y + nd.row0 + row + j0 * sl.ldy;
        ldy = kind == OZ_FINAL ? ldo : sl.ldy;
      } else {
        int64_t o;
        if (kind == OZ_UP_LEAF) o = nd.wz + row - nd.gm;
        else if (kind == OZ_UP_BRANCH)
          o = row < nd.kv ? nd.wz + row
                          : (row < nd.kv + nd.cku[0] ? nd.cwf[0] + row - nd.kv : nd.cwf[1] + row - nd.kv - nd.cku[0]);
        else o = row < nd.cku[0] ? nd.cwf[0] + row : nd.cwf[1] + row - nd.cku[0];
        ldo = sl.ldws;
        out = (double*)sl.ws + o + j0 * ldo;
        old = out;
        ldy = ldo;
        beta = kind == OZ_DOWN ? 1.0 : 0.0;
      }
      // bit tests: FP64 comparisons would go to the FP64 pipe
      const long long one = 0x3FF0000000000000ll, ab = __double_as_longlong(alpha), bb = __double_as_longlong(beta);
      const int mode = (bb << 1) == 0 ? (ab == one ? 0 : 1) : bb != one ? 4 : ab == one ? 2 : ab == (one | (1ll << 63)) ? 3 : 4;
      if (!waited) {
        asm volatile("griddepcontrol.wait;" ::: "memory");   // the previous step's outputs
        waited = true;
      }
      double acc[CW];
#pragma unroll
      for (int i = 0; i < CW; ++i) acc[i] = 0.0;
      const unsigned char* img = x.img;
      for (int c = 0; c * KC < x.K && ok; ++c, ++chunk) {
        const int kc = min(KC, x.K - c * KC), nst = (kc + KS - 1) / KS;
        const int ea = rin ? __ldg(reinterpret_cast<const int*>(img + (int64_t)nst * oz::kSlices * round8(x.rt) * 64) + lrow)
                           : oz::kZero;
        img += oz_chunk_bytes(x.rt, x.K, c);
        ok = __all_sync(0xffffffffu, wait_bar(&s_acc, chunk & 1, limit, &s_fail));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;");
        uint32_t direct = 0;
        const bool idle = !__any_sync(0xffffffffu, rin);   // no row of the tile in this warp
#pragma unroll
        for (int g = 0; g < CW / 4; ++g) {
          if (4 * g >= nc || idle) break;   // uniform over the warp
          __syncwarp();
          long long hi[4], lo[4];
          float sabs[4];
          oz::gather4<NC>(tacc + 4 * g, hi, lo, sabs);
          double d[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int eb = s_col[chunk & 3][cw0 + 4 * g + i];
            const bool fast = oz::in_range(ea, eb) && sabs[i] >= oz::kAbsMin;
            d[i] = fast ? oz::assemble(hi[i], lo[i], ea + eb - 2114) : 0.0;
            if (!fast && rin && 4 * g + i < nc && !oz::is_zero(ea, eb)) direct |= 1u << (4 * g + i);
          }
          if (c == 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[4 * g + i] = d[i];
          } else {
            asm volatile("");   // a branch: FP64 additions only where there is more than one chunk
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[4 * g + i] += d[i];
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncwarp();
        if (lane == 0) arrive(&s_read);
        // flagged outputs, summed by the warp, four terms per lane
        for (uint32_t rows = __ballot_sync(0xffffffffu, direct != 0); rows; rows &= rows - 1) {
          const int src = __ffs(rows) - 1;
          const uint32_t cols = __shfl_sync(0xffffffffu, direct, src);
          const int frow = x.t0 + 32 * (warp & 3) + src;
          double av[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int k = lane + 32 * q;
            av[q] = k < kc ? oz_entry(nd, kind, frow, c * KC + k) : 0.0;
          }
#pragma unroll
          for (int i = 0; i < CW; ++i) {
            if (!(cols >> i & 1)) continue;   // uniform over the warp
            double t = 0.0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int k = lane + 32 * q, kk = c * KC + k;
              if (k >= kc) continue;
              const int64_t j = j0 + i;
              double xv;
              if (kind == OZ_UP_LEAF) xv = sl.B[nd.col0 + kk + j * sl.ldb];
              else if (kind == OZ_UP_BRANCH)
                xv = ((const double*)sl.ws)[(kk < nd.ckv[0] ? nd.cwz[0] + kk : nd.cwz[1] + kk - nd.ckv[0]) + j * sl.ldws];
              else xv = ((const double*)sl.ws)[nd.wf + kk + j * sl.ldws];
              t = fma(av[q], xv, t);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            if (lane == src) acc[i] += t;
          }
        }
      }
      if (!ok || nc <= 0) continue;
      if (rin) {
        if (mode == 1) {
          asm volatile("");
#pragma unroll
          for (int i = 0; i < CW; ++i) acc[i] *= alpha;
        } else if (mode >= 2) {
          double y[CW];
#pragma unroll
          for (int i = 0; i < CW; ++i) y[i] = i < nc ? old[i * ldy] : 0.0;
          if (mode == 2) {
            asm volatile("");
#pragma unroll
            for (int i = 0; i < CW; ++i) acc[i] = y[i] + acc[i];
          } else if (mode == 3) {
            asm volatile("");
#pragma unroll
            for (int i = 0; i < CW; ++i) acc[i] = y[i] - acc[i];
          } else {
            asm volatile("");
#pragma unroll
            for (int i = 0; i < CW; ++i) acc[i] = fma(beta, y[i], alpha * acc[i]);
          }
        }
#pragma unroll
        for (int i = 0; i < CW; ++i)
          if (i < nc) out[i * ldo] = acc[i];
      }
      if (sl.colnorm2 != nullptr && (kind == OZ_FINAL || (kind == OZ_UP_LEAF && nd.root))) {
        // sums of squares over the warp's rows: halving the columns a lane holds
        // at every step (CW + 1 additions or a few more instead of 5 CW)
#pragma unroll
        for (int i = 0; i < CW; ++i) acc[i] = rin && i < nc ? acc[i] * acc[i] : 0.0;
        int first = 0;
#pragma unroll
        for (int w = CW / 2, o = 16; w >= 1; w >>= 1, o >>= 1) {
          const bool up = (lane & o) != 0;
#pragma unroll
          for (int i = 0; i < CW / 2; ++i) {
            if (i < w) {
              const double send = up ? acc[i] : acc[i + w], keep = up ? acc[i + w] : acc[i];
              acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
          }
          if (up) first += w;
        }
        constexpr int left = 32 / CW;   // lanes that still hold parts of the same column
#pragma unroll
        for (int o = left / 2; o >= 1; o >>= 1) acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
        if ((lane & (left - 1)) == 0 && first < nc) atomicAdd(sl.colnorm2 + j0 + first, acc[0]);
      }
    }
  }
  // in every block, units or not: the launch after this one waits for this grid only,
  // so a grid of empty units (a level of rank 0) must not end before the one before it
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(R::tmem));
  if (tid == 0 && s_fail)
    for (int64_t u = blockIdx.x; u < nunits; u += gridDim.x) {
      const Task tk = tasks[u / ((int64_t)nchunk * ntile)];
      if (slots[tk.slot].err) atomicCAS(slots[tk.slot].err, DEV_OK, DEV_TIMEOUT);
    }
}

template <int NC>
cudaError_t launch_nc(int kind, const Task* t, int64_t nt, const Slot* s, int rmax, int rows, int sms, cudaStream_t st) {
  static SmemOptIn opt_in;
  const cudaError_t e = opt_in((const void*)ozmv_kernel<NC>, Ring<NC>::smem);
  if (e != cudaSuccess) return e;
  const int nchunk = (rmax + NC - 1) / NC, ntile = std::max(1, (rows + TR - 1) / TR);
  const int64_t units = nt * nchunk * ntile;
  const uint32_t polls = pmv_poll_limit();
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)std::min<int64_t>(units, sms));
  cfg.blockDim = dim3(OT);
  cfg.dynamicSmemBytes = Ring<NC>::smem;
  cfg.stream = st;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = kind == OZ_UP_LEAF ? 0 : 1;   // the first step waits for whatever came before
  return cudaLaunchKernelEx(&cfg, ozmv_kernel<NC>, t, units, ntile, nchunk, s, kind, polls ? polls : 1u << 22);
}

}  // namespace

int64_t ozmv_image_bytes(const Node& nd, bool up) {
  const int kind = up ? (nd.leaf ? OZ_UP_LEAF : OZ_UP_BRANCH) : (nd.leaf ? OZ_FINAL : OZ_DOWN);
  const int rows = oz_rows(nd, kind), K = oz_inner(nd, kind);
  int64_t b = (int64_t)(rows / TR) * oz_tile_bytes(TR, K);
  if (rows % TR) b += oz_tile_bytes(rows % TR, K);
  return b;
}

cudaError_t launch_ozmv_prep(int kind, const Task* t, int64_t nt, int rows, int inner, unsigned char* base,
                             cudaStream_t st) {
  if (nt <= 0 || rows <= 0 || inner <= 0) return cudaSuccess;
  static SmemOptIn opt_in;
  const cudaError_t e = opt_in((const void*)ozmv_prep_kernel, kPrepSmem);
  if (e != cudaSuccess) return e;
  const int ntile = (rows + TR - 1) / TR, nchunk = (inner + KC - 1) / KC;
  if (nt * ntile * nchunk > INT32_MAX) return cudaErrorInvalidValue;
  ozmv_prep_kernel<<<(unsigned)(nt * ntile * nchunk), PT, kPrepSmem, st>>>(t, kind, ntile, nchunk, base);
  return cudaGetLastError();
}

cudaError_t launch_ozmv(int kind, const Task* t, int64_t nt, const Slot* s, int rmax, int rows, int sms, cudaStream_t st) {
  if (nt <= 0 || rmax <= 0) return cudaSuccess;
  // 16 columns per unit while that leaves SMs idle: the units of a small level
  // are its latency
  const int64_t wide = nt * std::max(1, (rows + TR - 1) / TR) * ((rmax + 31) / 32);
  return rmax <= 16 || 2 * wide <= sms ? launch_nc<16>(kind, t, nt, s, rmax, rows, sms, st)
                                       : launch_nc<32>(kind, t, nt, s, rmax, rows, sms, st);
}

}  // namespace hss
