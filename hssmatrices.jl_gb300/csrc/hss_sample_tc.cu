// The dense sample products S = A Omega, S = A^T Omega of randomized compression
// (reference src/compression.jl:290-291, :326-327, :336-337) in FP64 accuracy on
// the tensor cores (hss_oz.cuh): GB300's FP64 pipe needs 64 clocks per warp
// instruction, so the products were bound by it (93 % of its peak) and not by
// the bytes of A; as 45 exact bf16 digit products they come within a small
// factor of the time that reading A takes.
//
// oz_prep_kernel cuts Omega (k x r, small) into digit slices once per call, in
// the operand layout, per chunk of 128 rows and tile of NC columns.
// sample_tc_kernel runs one block per (128 rows of op(A), a range of chunks,
// column tile): 512 threads hold a 128 x 128 chunk of A in registers (32 values
// each), find the row exponents, and cut it in four stages of K = 32 into the
// two halves of a shared-memory ring while the next chunk's loads go out as the
// registers empty; one thread issues the stage's MMAs (M = 128, N up to 256: a
// digit of A against several digits of Omega at once).  After four stages the
// accumulators are put together and added to FP64 sums in registers, the only
// FP64 instructions (one addition per output and chunk).  A thread keeps at most
// 32 + NC / 4 doubles in registers, which with 512 threads is what the register
// file holds; the ring (184 KB, with tiles of 32 columns 200 KB) leaves one block per SM.
//
// What bounds it now: cutting A into digits, about 45 integer instructions per
// entry (ALU pipe 52 % busy, tensor pipe 20 %, DRAM 17 %); per chunk of 128 x 128
// about 12 us.  Measured (one GB300, L2 cold): 8192 x 8192, 30 columns 3750 ->
// 444 us; 16384 x 16384, 20 columns 9500 -> 1380 us (1.55 TB/s of A); 4096 x
// 4096, 20 columns 604 -> 122 us.  Error against exact sums of 4096 terms, root
// mean square relative to the sums, in units of roundoff: 4.8 -> 1.2 (a kernel matrix),
// 4.0 -> 1.3 (normal entries).
//
// Blocks of one row tile split the chunks so that every SM has work; their sums
// go to a scratch buffer that sample_reduce_kernel adds in a fixed order.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "hss_oz.cuh"
#include "hss_internal.h"
#include "hss_optin.h"
#include "hss_sample.h"

namespace hss {

namespace {

constexpr int ST = 512;           // threads
constexpr int SM_ = 128;          // rows per block
constexpr int KC = 128;           // K per chunk
constexpr int KS = 32;            // K per stage
constexpr int kASlice = SM_ * KS * 2;   // bytes of one slice of a stage of A: 8 KB

template <int NC>
struct Sizes {
  static constexpr int bslice = NC * KS * 2;                 // bytes of one slice of a stage of Omega
  static constexpr int bstage = oz::kSlices * bslice;
  static constexpr int bchunk = 4 * bstage + NC * 4;         // four stages, then the column codes
  static constexpr int stage = oz::kSlices * kASlice + bstage;
  static constexpr int smem = 2 * stage;
  static constexpr uint32_t tmem = NC == 32 ? 512 : 256;     // (kAcc + 1) NC columns, a power of two
};

// One block per (chunk, column tile): codes and slices of X(k0 .. k0 + 127, c0 .. c0 + NC - 1).
template <int NC>
__global__ void __launch_bounds__(NC * 16) oz_prep_kernel(const double* __restrict__ X, int64_t ldx, int64_t k,
                                                          int64_t r, unsigned char* __restrict__ out) {
  const int kg = threadIdx.x & 15, c = threadIdx.x >> 4;     // 16 threads per column, 8 rows each
  const int64_t col = (int64_t)blockIdx.y * NC + c, k0 = (int64_t)blockIdx.x * KC + 8 * kg;
  unsigned char* reg = out + ((int64_t)blockIdx.y * gridDim.x + blockIdx.x) * Sizes<NC>::bchunk;
  unsigned long long b[8];
  uint32_t hmax = 0, have = 0;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    b[e] = (col < r && k0 + e < k) ? oz::bits_of(__ldg(X + k0 + e + col * ldx)) : 0ull;
    oz::scan(b[e], hmax, have);
  }
  int emax = (int)(hmax >> 20);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) {
    emax = max(emax, __shfl_xor_sync(0xffffffffu, emax, o));
    have |= __shfl_xor_sync(0xffffffffu, have, o);
  }
  if (kg == 0) reinterpret_cast<int*>(reg + 4 * Sizes<NC>::bstage)[c] = oz::exp_code(emax, have != 0);
  uint4 w[oz::kSlices];
  uint32_t* ww = reinterpret_cast<uint32_t*>(w);
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    const oz::Pair pr(b[2 * h], b[2 * h + 1], emax);
#pragma unroll
    for (int p = 0; p < oz::kDigits; ++p) ww[4 * p + h] = pr.digit(p);
    ww[4 * oz::kDigits + h] = pr.top_abs();
  }
  unsigned char* dst = reg + (kg >> 2) * Sizes<NC>::bstage + oz::core_off(c, kg & 3);
#pragma unroll
  for (int p = 0; p < oz::kSlices; ++p) *reinterpret_cast<uint4*>(dst + p * Sizes<NC>::bslice) = w[p];
}

struct TcProblem {
  const double* A;
  int64_t lda;
  const double* X;
  int64_t ldx;
  double* Y;
  int64_t ldy;
  int64_t m, k, r;
  int64_t per;              // chunks per block along z
  const unsigned char* xs;  // slices of X
  double alpha, beta;
  double* partial;          // null: Y = alpha acc + beta Y
  uint32_t limit;           // polls of a wait before it gives up
  int32_t* status;          // gets DEV_TIMEOUT then
};

// TRANS: op(A) = A^T, rows of op(A) are columns of A.  Thread layouts of a
// chunk: plain, row = tid % 128 and the K group of 8 in every stage tid / 128
// (consecutive lanes read consecutive rows); transposed, row = 8 warp + lane / 4
// and K pairs 2 (lane % 4) of each of the stage's four K groups (four lanes
// read 64 consecutive bytes of a column).
template <int NC, bool TRANS>
__global__ void __launch_bounds__(ST, 1) sample_tc_kernel(TcProblem p) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ uint32_t s_tmem;
  __shared__ __align__(8) uint64_t s_full[2], s_done[2];   // a stage's slices of Omega are in; its MMAs are done
  __shared__ int s_code[4][SM_];
  __shared__ int s_row[SM_], s_col[NC];
  using Z = Sizes<NC>;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t row0 = (int64_t)blockIdx.x * SM_;
  const int64_t nchunk = (p.k + KC - 1) / KC;
  const int64_t c0 = (int64_t)blockIdx.z * p.per, c1 = min(nchunk, c0 + p.per);
  const unsigned char* xs = p.xs + (int64_t)blockIdx.y * nchunk * Z::bchunk;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(oz::smem_u32(&s_tmem)),
                 "r"(Z::tmem));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      oz::mbar_init(&s_full[i]);
      oz::mbar_init(&s_done[i]);
    }
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = s_tmem;

  const int lr = TRANS ? 8 * warp + (lane >> 2) : tid & (SM_ - 1);   // row within the tile
  const int64_t row = row0 + lr;
  // value e of stage s of a chunk is at K offset KS s + koff(e); rows beyond m
  // read row m - 1 (their results are not stored)
  auto koff = [&](int e) -> int { return TRANS ? 8 * (e >> 1) + 2 * (lane & 3) + (e & 1) : 8 * (tid >> 7) + e; };
  const double* arow = TRANS ? p.A + min(row, p.m - 1) * p.lda : p.A + min(row, p.m - 1);
  const int64_t kstep = TRANS ? 1 : p.lda;
  double v[4][8];
  auto load = [&](int64_t c, int s) {
    const int64_t kb = c * KC + KS * s;
    if (c < c1 && kb + KS <= p.k) {
      const double* q = arow + (kb + koff(0)) * kstep;
      if constexpr (TRANS) {
#pragma unroll
        for (int e = 0; e < 8; ++e) v[s][e] = __ldg(q + 8 * (e >> 1) + (e & 1));
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e, q += kstep) v[s][e] = __ldg(q);
      }
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int64_t kk = kb + koff(e);
        v[s][e] = (c < c1 && kk < p.k) ? __ldg(arow + kk * kstep) : 0.0;
      }
    }
  };
#pragma unroll
  for (int s = 0; s < 4; ++s) load(c0, s);

  double acc[NC / 4];
#pragma unroll
  for (int i = 0; i < NC / 4; ++i) acc[i] = 0.0;
  // output mapping: rows 32 (warp % 4) + lane, columns (NC / 4) (warp / 4) ..
  const int orow = 32 * (warp & 3) + lane, oc0 = (NC / 4) * (warp >> 2);
  const int64_t ncol = min((int64_t)NC, p.r - (int64_t)blockIdx.y * NC);
  const uint32_t tacc = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)oc0;

  uint32_t use = 0;   // stages issued so far: ring half use & 1, its use / 2-th use
  uint32_t loads = 0, mmas = 0;   // (thread 0) copies and groups of MMAs issued
  // A wait that runs out makes `fail` true in its thread; nothing is issued after it, and
  // the block leaves together at the next barrier.
  bool fail = false, ok = true;
  for (int64_t c = c0; c < c1 && ok; ++c) {
    // row exponents of the chunk
    uint32_t hmax = 0, have = 0;
#pragma unroll
    for (int s = 0; s < 4; ++s)
#pragma unroll
      for (int e = 0; e < 8; ++e) oz::scan(oz::bits_of(v[s][e]), hmax, have);
    int emax = (int)(hmax >> 20);
    if constexpr (TRANS) {
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) {
        emax = max(emax, __shfl_xor_sync(0xffffffffu, emax, o));
        have |= __shfl_xor_sync(0xffffffffu, have, o);
      }
      if ((lane & 3) == 0) s_row[lr] = oz::exp_code(emax, have != 0);
      if (tid < NC) s_col[tid] = reinterpret_cast<const int*>(xs + c * Z::bchunk + 4 * Z::bstage)[tid];
    } else {
      s_code[tid >> 7][lr] = emax | (have ? 1 << 16 : 0);
      if (tid < NC) s_col[tid] = reinterpret_cast<const int*>(xs + c * Z::bchunk + 4 * Z::bstage)[tid];
      __syncthreads();
      have = 0;
      emax = 0;
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const int w = s_code[g][lr];
        emax = max(emax, w & 0xFFFF);
        have |= w >> 16;
      }
      if (tid < SM_) s_row[lr] = oz::exp_code(emax, have != 0);
    }

#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int h = use & 1;
      unsigned char* abuf = smem + h * Z::stage;
      unsigned char* bbuf = abuf + oz::kSlices * kASlice;
      if (!ok) continue;
      // the ring half is free once the MMAs of its previous use are done
      if (use >= 2) fail = fail || !oz::mbar_wait(&s_done[h], ((use >> 1) - 1) & 1, p.limit);
      if (tid == 0 && !fail) {
        oz::bulk_load(bbuf, xs + c * Z::bchunk + s * Z::bstage, Z::bstage, &s_full[h]);
        ++loads;
      }
      if constexpr (TRANS) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const oz::Pair pr(oz::bits_of(v[s][2 * u]), oz::bits_of(v[s][2 * u + 1]), emax);
          unsigned char* dst = abuf + oz::core_off(lr, u) + 4 * (lane & 3);
#pragma unroll
          for (int q = 0; q < oz::kDigits; ++q) *reinterpret_cast<uint32_t*>(dst + q * kASlice) = pr.digit(q);
          *reinterpret_cast<uint32_t*>(dst + oz::kDigits * kASlice) = pr.top_abs();
        }
      } else {
        const oz::Pair p0(oz::bits_of(v[s][0]), oz::bits_of(v[s][1]), emax);
        const oz::Pair p1(oz::bits_of(v[s][2]), oz::bits_of(v[s][3]), emax);
        const oz::Pair p2(oz::bits_of(v[s][4]), oz::bits_of(v[s][5]), emax);
        const oz::Pair p3(oz::bits_of(v[s][6]), oz::bits_of(v[s][7]), emax);
        unsigned char* dst = abuf + oz::core_off(lr, tid >> 7);
#pragma unroll
        for (int q = 0; q < oz::kDigits; ++q)
          *reinterpret_cast<uint4*>(dst + q * kASlice) = make_uint4(p0.digit(q), p1.digit(q), p2.digit(q), p3.digit(q));
        *reinterpret_cast<uint4*>(dst + oz::kDigits * kASlice) =
            make_uint4(p0.top_abs(), p1.top_abs(), p2.top_abs(), p3.top_abs());
      }
      load(c + 1, s);   // the next chunk's values replace the ones just used
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;");
      ok = !__syncthreads_or(fail);
      if (!ok) continue;
      if (tid == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;");
        fail = !oz::mbar_wait(&s_full[h], (use >> 1) & 1, p.limit);
        if (!fail) {
          oz::stage_mma<SM_, NC>(tmem, oz::smem_u32(abuf), kASlice, oz::smem_u32(bbuf), s == 0);
          oz::mma_commit(&s_done[h]);
          ++mmas;
        }
      }
      ++use;
    }
    if (!ok) break;
    // all MMAs of the chunk are done when its last stage's are
    const uint32_t last = use - 1;
    fail = fail || !oz::mbar_wait(&s_done[last & 1], (last >> 1) & 1, p.limit);
    asm volatile("tcgen05.fence::after_thread_sync;");
    const int ea = s_row[orow];
    uint32_t direct = 0;   // columns of this thread's row that are summed in FP64
#pragma unroll
    for (int g = 0; g < NC / 16; ++g) {
      if (oc0 + 4 * g >= ncol) break;   // uniform over the warp
      long long hi[4], lo[4];
      float sabs[4];
      oz::gather4<NC>(tacc + 4 * g, hi, lo, sabs);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int cc = oc0 + 4 * g + i;
        const int eb = s_col[cc];
        if (cc >= ncol || row0 + orow >= p.m || oz::is_zero(ea, eb)) continue;
        if (oz::in_range(ea, eb) && sabs[i] >= oz::kAbsMin)
          acc[4 * g + i] += oz::assemble(hi[i], lo[i], ea + eb - 2114);
        else
          direct |= 1u << (4 * g + i);
      }
    }
    __syncwarp();
    // the warp sums the flagged outputs row by row, four terms per lane
    for (uint32_t rows = __ballot_sync(0xffffffffu, direct != 0); rows; rows &= rows - 1) {
      const int src = __ffs(rows) - 1;
      const uint32_t cols = __shfl_sync(0xffffffffu, direct, src);
      const int64_t grow = row0 + 32 * (warp & 3) + src, kb = c * KC + lane;
      const double* a = TRANS ? p.A + grow * p.lda : p.A + grow;
      double av[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) av[q] = kb + 32 * q < p.k ? __ldg(a + (kb + 32 * q) * kstep) : 0.0;
#pragma unroll
      for (int i = 0; i < NC / 4; ++i) {
        if (!(cols >> i & 1)) continue;   // uniform over the warp
        const double* x = p.X + ((int64_t)blockIdx.y * NC + oc0 + i) * p.ldx + kb;
        double t = 0.0;
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (kb + 32 * q < p.k) t = fma(av[q], __ldg(x + 32 * q), t);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == src) acc[i] += t;
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    ok = !__syncthreads_or(fail);   // the accumulators and the codes may be overwritten
    asm volatile("tcgen05.fence::after_thread_sync;");
  }

  if (row0 + orow < p.m) {
#pragma unroll
    for (int i = 0; i < NC / 4; ++i) {
      if (!ok) acc[i] = __longlong_as_double(0x7FF8000000000000ll);   // a wait ran out: NaN
      const int64_t gi = row0 + orow, gj = (int64_t)blockIdx.y * NC + oc0 + i;
      if (gj >= p.r) continue;
      if (p.partial) {
        p.partial[(int64_t)blockIdx.z * p.m * p.r + gi + gj * p.m] = acc[i];
      } else {
        double* y = p.Y + gi + gj * p.ldy;
        *y = p.beta == 0.0 ? p.alpha * acc[i] : fma(p.alpha, acc[i], p.beta * *y);
      }
    }
  }
  if (!ok && tid == 0) {
    if (p.status) *(volatile int32_t*)p.status = DEV_TIMEOUT;
    __threadfence_system();
    // copies and MMAs that may still be running end before the block does (bounded)
    for (uint32_t i = loads > 2 ? loads - 2 : 0; i < loads; ++i) oz::mbar_wait(&s_full[i & 1], (i >> 1) & 1);
    for (uint32_t i = mmas > 2 ? mmas - 2 : 0; i < mmas; ++i) oz::mbar_wait(&s_done[i & 1], (i >> 1) & 1);
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(Z::tmem));
}

template <int NC>
cudaError_t launch_tc(TcProblem p, int trans, const SampleTcPlan& pl, unsigned char* xs, cudaStream_t st) {
  const int64_t nchunk = (p.k + KC - 1) / KC;
  const unsigned tiles = (unsigned)((p.r + NC - 1) / NC);
  static SmemOptIn opt_in[2];
  auto* kernel = trans ? sample_tc_kernel<NC, true> : sample_tc_kernel<NC, false>;
  const cudaError_t e = opt_in[trans ? 1 : 0]((const void*)kernel, Sizes<NC>::smem);
  if (e != cudaSuccess) return e;
  if (nchunk > 0) oz_prep_kernel<NC><<<dim3((unsigned)nchunk, tiles), NC * 16, 0, st>>>(p.X, p.ldx, p.k, p.r, xs);
  const dim3 grid((unsigned)((p.m + SM_ - 1) / SM_), tiles, (unsigned)pl.nsplit);
  kernel<<<grid, ST, Sizes<NC>::smem, st>>>(p);
  return cudaGetLastError();
}

}  // namespace

SampleTcPlan sample_tc_plan(int64_t m, int64_t k, int64_t r, int sms) {
  SampleTcPlan pl;
  pl.nc = r <= 16 ? 16 : 32;
  const int64_t nchunk = (k + KC - 1) / KC, tiles = (r + pl.nc - 1) / pl.nc;
  const int64_t blocks = (m + SM_ - 1) / SM_ * tiles;
  // the split with the shortest schedule: rounds of one block per SM, each as
  // long as its chunks and about one more (start, first loads, output)
  int64_t best = INT64_MAX;
  for (int64_t z = 1; z <= std::min<int64_t>(std::max<int64_t>(nchunk, 1), 64); ++z) {
    const int64_t per = (nchunk + z - 1) / z, cost = (blocks * z + sms - 1) / sms * (per + 1);
    if (cost < best) {
      best = cost;
      pl.per = per;
    }
  }
  pl.per = std::max<int64_t>(pl.per, 1);
  pl.nsplit = (int)std::max<int64_t>(1, (nchunk + pl.per - 1) / pl.per);
  const size_t bchunk = pl.nc == 16 ? Sizes<16>::bchunk : Sizes<32>::bchunk;
  pl.slice_bytes = ((size_t)tiles * nchunk * bchunk + 255) & ~size_t(255);
  pl.scratch_bytes = pl.slice_bytes + (pl.nsplit > 1 ? (size_t)pl.nsplit * m * r * sizeof(double) : 0);
  return pl;
}

cudaError_t launch_sample_tc(const double* A, int64_t lda, int64_t m, int64_t k, int trans, const double* X,
                             int64_t ldx, int64_t r, double* Y, int64_t ldy, double alpha, double beta,
                             const SampleTcPlan& pl, unsigned char* scratch, uint32_t limit, int32_t* status,
                             cudaStream_t st) {
  double* partial = pl.nsplit > 1 ? (double*)(scratch + pl.slice_bytes) : nullptr;
  const TcProblem p{A, lda, X, ldx, Y, ldy, m, k, r, pl.per, scratch, alpha, beta, partial, limit, status};
  cudaError_t e = pl.nc == 16 ? launch_tc<16>(p, trans, pl, scratch, st) : launch_tc<32>(p, trans, pl, scratch, st);
  if (e == cudaSuccess && partial) e = launch_sample_reduce(partial, pl.nsplit, m, r, Y, ldy, alpha, beta, st);
  return e;
}

}  // namespace hss
