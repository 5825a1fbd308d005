// ULV solve kernels with the right-hand sides held in registers.
//
// One thread block per tree node; a group of TPC consecutive lanes owns one
// right-hand-side column, lane gl holding rows gl, gl+TPC, gl+2*TPC, ... (up
// to MR rows).  Reflector applications are group dot products (shuffle
// reductions inside the group) followed by register updates; the triangular
// solves broadcast each solved entry from its owner lane.  No block-wide
// barrier sits inside the sequential sweeps.
//
// A level is bound by one block's chain, a list of many blocks by the FP64 pipe:
// * a division is about forty FP64 instructions of 64 clocks on the chain of every
//   row of a substitution; the diagonal's reciprocals are formed once per block
//   instead, and a quotient is a product and one correction (a finished column is
//   looked over for entries that this fails, and done again by divisions then; a test
//   per row cost 1.2 % of a resident solve and 2.3 % of a mixed batch, this 0.3 %);
// * 8 lanes per right-hand side (four per warp) spend 20 FP64 instructions on a
//   reflector of 64 rows for four right-hand sides, 32 lanes 10 for one: FP64
//   lists longer than two rounds of the SMs take 8 lanes, shorter ones 32;
// * a launch after the first of a sweep starts while the level before it ends
//   (programmatic dependent launch) and copies its factor blocks meanwhile.
// Measured (one GB300, CUDA events around each launch): n = 65536, k = 32, 32
// right-hand sides in FP64, leaf level upward 2540 -> 1225 us and downward 1565 ->
// 983, 256-node level upward 541 -> 295, root 72 -> 45; 1200 unknowns, k = 16 in
// FP64, a level upward 50 -> 34 us.  FP32, 64 x 64 nodes: upward 26.6 -> 20.5 us a
// level (16-byte-stride copies without index divisions, no transposed stores), with
// the overlap of consecutive levels a resident solve of n = 16384 with 4
// right-hand sides 1020 -> 773 us.
//
// Upward pass per node (reference src/ulvfactor.jl:22-57, :74, :89):
//   b = rhs rows (leaf) or [b1; b2] - [T12 u2; T21 u1] (branch)
//   b <- Q_ql^T b;  zloc = L1 \ b[0:mk];  b_red = b[mk:m] - L2 zloc;
//   u = V[0:mk,:]^T zloc (+ W1^T u1 + W2^T u2);  x[0:mk] = zloc;
//   root: x = LU \ b (src/ulvfactor.jl:83).
// Downward pass per node (src/ulvfactor.jl:98-107): x <- Q_lq^T x, then the
// un-eliminated tail goes to the children (or the output at a leaf).
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include "hss_factor.cuh"
#include "hss_internal.h"
#include "hss_launch.h"
#include "hss_optin.h"

namespace hss {

namespace {

constexpr int ST = 256;

// The launch's dependents may be scheduled; wait for the launch it depends on.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// dst (ld ldd) = rows x cols block of src (ld lds), a column per warp; tril: rows
// from the diagonal on only.
template <typename T>
__device__ __forceinline__ void stage_block(T* dst, int ldd, const T* src, int64_t lds, int rows, int cols, bool tril = false);

// Asynchronous element copy global -> shared (cp.async, 4 or 8 bytes): the
// staging copies of a block are all in flight at once; cpa_wait() waits for
// this thread's copies, a barrier then publishes everyone's.  The sources
// (factor blocks, the previous level's workspace) do not change during the
// launch.
template <typename T>
__device__ __forceinline__ void cpa(T* s, const T* g) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(s);
  if constexpr (sizeof(T) == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(sa), "l"(g) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sa), "l"(g) : "memory");
}
__device__ __forceinline__ void cpa_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <typename T>
__device__ __forceinline__ void stage_block(T* dst, int ldd, const T* src, int64_t lds, int rows, int cols, bool tril) {
  const int lane = threadIdx.x & 31;
  for (int c = threadIdx.x >> 5; c < cols; c += ST / 32)
    for (int i = lane + (tril ? c & ~31 : 0); i < rows; i += 32) cpa(dst + i + c * ldd, src + i + (int64_t)c * lds);
}

template <int TPC, typename T>
__device__ __forceinline__ T gsum(T v) {
#pragma unroll
  for (int o = TPC / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, TPC);
  return v;
}

// Forward substitution L x = b in registers (L lower, ld ldl, size nr; rd: the
// reciprocals of its diagonal).
template <typename T, int TPC, int RPT, bool UNIT>
__device__ __forceinline__ void lower_solve(T (&b)[RPT], const T* __restrict__ L, int ldl, int nr, int gl, const T* rd) {
#pragma unroll
  for (int s = 0; s < RPT; ++s) {
    if (s * TPC >= nr) break;
    for (int o = 0; o < TPC; ++o) {
      const int c = s * TPC + o;
      if (c >= nr) break;
      const T bc = __shfl_sync(0xffffffffu, b[s], o, TPC);
      const T xc = UNIT ? bc : fac::quot(bc, L[c + (int64_t)c * ldl], rd[c]);
      if (gl == o) b[s] = xc;
#pragma unroll
      for (int s2 = s; s2 < RPT; ++s2) {
        const int row = gl + s2 * TPC;
        if (row > c && row < nr) b[s2] -= L[row + (int64_t)c * ldl] * xc;
      }
    }
  }
}

// Backward substitution U x = b (U upper, non-unit).
template <typename T, int TPC, int RPT>
__device__ __forceinline__ void upper_solve(T (&b)[RPT], const T* __restrict__ A, int lda, int nr, int gl, const T* rd) {
#pragma unroll
  for (int s = RPT - 1; s >= 0; --s) {
    if (s * TPC >= nr) continue;
    for (int o = TPC - 1; o >= 0; --o) {
      const int c = s * TPC + o;
      if (c >= nr) continue;
      const T bc = __shfl_sync(0xffffffffu, b[s], o, TPC);
      const T xc = fac::quot(bc, A[c + (int64_t)c * lda], rd[c]);
      if (gl == o) b[s] = xc;
#pragma unroll
      for (int s2 = 0; s2 <= s; ++s2) {
        const int row = gl + s2 * TPC;
        if (row < c) b[s2] -= A[row + (int64_t)c * lda] * xc;
      }
    }
  }
}

// Whether a solution in registers holds an entry that quot failed (L: the block whose
// diagonal it was divided by).
template <typename T, int TPC, int RPT>
__device__ __forceinline__ bool failed(const T (&b)[RPT], const T* __restrict__ L, int ld, int nr, int gl) {
  bool bad = false;
#pragma unroll
  for (int s = 0; s < RPT; ++s) {
    const int row = gl + s * TPC;
    if (row < nr) bad = bad || fac::quot_failed(b[s], L[row + (int64_t)row * ld]);
  }
  return bad;
}

// The same steps by divisions, on a column in shared memory, for right-hand sides that
// the reciprocals failed (entries that are infinite, NaN or out of range): every warp
// that calls takes all its columns through them.
template <typename T, int TPC>
__device__ __noinline__ void reflect_slow(T* col, const T* U, int ldU, const T* tq, int m, int k, int mk, int gl) {
  for (int c = k - 1; c >= 0; --c) {
    const int p = mk + c;
    T d = T(0);
    for (int row = gl; row <= p; row += TPC) d += (row == p ? T(1) : U[row + (int64_t)c * ldU]) * col[row];
    d = gsum<TPC>(d) * tq[c];
    for (int row = gl; row <= p; row += TPC) col[row] -= d * (row == p ? T(1) : U[row + (int64_t)c * ldU]);
    __syncwarp();
  }
}
template <typename T, int TPC>
__device__ __noinline__ void lower_slow(T* col, const T* L, int ldl, int nr, int gl, bool unit) {
  for (int c = 0; c < nr; ++c) {
    const T x = unit ? col[c] : col[c] / L[c + (int64_t)c * ldl];
    __syncwarp();
    if (gl == 0) col[c] = x;
    for (int row = c + 1 + gl; row < nr; row += TPC) col[row] -= L[row + (int64_t)c * ldl] * x;
    __syncwarp();
  }
}
template <typename T, int TPC>
__device__ __noinline__ void upper_slow(T* col, const T* A, int lda, int nr, int gl) {
  for (int c = nr - 1; c >= 0; --c) {
    const T x = col[c] / A[c + (int64_t)c * lda];
    __syncwarp();
    if (gl == 0) col[c] = x;
    for (int row = gl; row < c; row += TPC) col[row] -= A[row + (int64_t)c * lda] * x;
    __syncwarp();
  }
}

// Elements of shared memory the upward kernel stages for one node (beyond the
// right-hand sides); the host sizes launches with the level's largest value.
__host__ __device__ inline int64_t solve_up_stage_elems(int m, int k, int mk, int nk, int kv, bool leaf, bool root,
                                                       int mr1, int mr2, int kv1, int kv2, int cpb) {
  int64_t e = 0;
  if (root) e += (int64_t)m * m;
  else if (mk > 0) e += (int64_t)m * k + (int64_t)mk * mk + (int64_t)k * nk + (int64_t)(nk | 1) * kv;
  if (!leaf) {
    e += (int64_t)mr1 * kv2 + (int64_t)mr2 * kv1 + (int64_t)(kv1 + kv2) * cpb;
    if (!root) e += (int64_t)((kv1 | 1) + (kv2 | 1)) * kv;
  }
  return e;
}

template <typename T, int TPC, int MR>
__global__ void __launch_bounds__(ST, sizeof(T) == 4 && MR > 64 ? 4 : MR / TPC > 8 ? 2 : 3) ulv_solve_up_reg(const Task* __restrict__ tasks,
                                                       const Slot* __restrict__ slots, int64_t stage_cap,
                                                       int nchunk) {
  constexpr int RPT = MR / TPC;
  constexpr int CPB = ST / TPC;
  constexpr int LDS = MR + 1;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ T s_rd[MR];      // reciprocals of the diagonal that is solved with
  T* sb = (T*)smraw;          // LDS x CPB right-hand sides
  T* sx = sb + LDS * CPB;     // staged operands
  pdl_trigger();
  const Task tk = tasks[blockIdx.x / nchunk];
  const int jchunk = (blockIdx.x % nchunk) * CPB;   // this block's columns: jchunk .. jchunk+CPB-1
  const Node* nodes = tk.nodes;
  const Node& nd = nodes[tk.node];
  const Slot& sl = slots[tk.slot];
  T* ws = (T*)sl.ws;
  const int64_t ld = sl.ldws;
  const T* fb = (const T*)sl.fbase;
  const int m = nd.m, n = nd.n, kv = nd.kv, r = sl.r;
  if (jchunk >= r) {
    pdl_wait();
    return;
  }
  const int tid = threadIdx.x, g = tid / TPC, gl = tid % TPC;
  const int k = nd.k, mk = nd.mk, nk = nd.nk;
  T* u = ws + nd.wu;
  const Node* c1 = nd.leaf ? nullptr : &nodes[nd.left];
  const Node* c2 = nd.leaf ? nullptr : &nodes[nd.right];
  const int mr1 = c1 ? c1->mr : 0, mr2 = c2 ? c2->mr : 0, kv1 = c1 ? c1->kv : 0, kv2 = c2 ? c2->kv : 0;
  const bool staged = solve_up_stage_elems(m, k, mk, nk, kv, nd.leaf, nd.root, mr1, mr2, kv1, kv2, CPB) <= stage_cap;

  // Every factor / generator block an inner loop reads is copied on chip once
  // (bulk, coalesced), unless the level's blocks do not fit: then they are
  // read from global memory in place.  Leading dimensions follow the copy.
  const T* Up = fb + nd.fU;  int ldU = m;       // QL reflectors m x k
  const T* Lp = fb + nd.fD;  int ldL = m;       // L1 (mk x mk) or the root LU (m x m)
  const T* L2p = fb + nd.fD + mk;  int ldL2 = m;      // L2[:, 0:nk], k x nk
  const T* Vap = fb + nd.fV; int ldVa = n;      // V[0:nk, :], nk x kv
  const T* T12p = nd.leaf ? nullptr : fb + nd.fT12;   // mr1 x kv2
  const T* T21p = nd.leaf ? nullptr : fb + nd.fT21;   // mr2 x kv1
  T* sW1 = nullptr;  T* sW2 = nullptr;  T* su1 = nullptr;  T* su2 = nullptr;
  int ldW1 = 0, ldW2 = 0;
  if (staged) {
    T* p = sx;
    if (nd.root) {
      stage_block(p, m, Lp, m, m, m);
      Lp = p; ldL = m; p += m * m;
    } else if (mk > 0) {
      stage_block(p, m, Up, m, m, k);
      Up = p; ldU = m; p += m * k;
      stage_block(p, mk, Lp, m, mk, mk, true);
      Lp = p; ldL = mk; p += mk * mk;
      stage_block(p, k, L2p, m, k, nk);
      L2p = p; ldL2 = k; p += k * nk;
      ldVa = nk | 1;   // odd: consecutive threads read consecutive columns
      stage_block(p, ldVa, Vap, n, nk, kv);
      Vap = p; p += ldVa * kv;
    }
    if (!nd.leaf) {
      stage_block(p, mr1, T12p, mr1, mr1, kv2);
      T12p = p; p += mr1 * kv2;
      stage_block(p, mr2, T21p, mr2, mr2, kv1);
      T21p = p; p += mr2 * kv1;
      if (!nd.root) {
        ldW1 = kv1 | 1; ldW2 = kv2 | 1;
        sW1 = p; p += ldW1 * kv;
        sW2 = p; p += ldW2 * kv;
        // (converted from the FP64 generators: register loads, eight in flight per lane)
        auto stage_w = [&](T* dst, int ldd, const double* src, int kc) {
          const int lane = tid & 31;
          for (int c0 = tid >> 5; c0 < kv; c0 += 8 * (ST / 32))
            for (int i = lane; i < kc; i += 32) {
              double w[8];
#pragma unroll
              for (int q = 0; q < 8; ++q)
                w[q] = c0 + q * (ST / 32) < kv ? __ldg(src + i + (int64_t)(c0 + q * (ST / 32)) * kc) : 0.0;
#pragma unroll
              for (int q = 0; q < 8; ++q)
                if (c0 + q * (ST / 32) < kv) dst[i + (c0 + q * (ST / 32)) * ldd] = (T)w[q];
            }
        };
        stage_w(sW1, ldW1, nd.W1, kv1);
        stage_w(sW2, ldW2, nd.W2, kv2);
      }
      su1 = p; p += kv1 * CPB;
      su2 = p; p += kv2 * CPB;
    }
  }
  // (from the factor storage itself: the staged copy is still on its way)
  for (int i = tid; i < (nd.root ? m : mk); i += ST) s_rd[i] = fac::recip(fb[nd.fD + i + (int64_t)i * m]);
  pdl_wait();   // what follows reads the level before
  for (int j0 = jchunk; j0 < jchunk + CPB && j0 < r; j0 += CPB) {
    const int ncol = min(CPB, r - j0);
    // ---- gather b for this chunk of columns into shared memory
    if (nd.leaf) {
      for (int e = tid; e < m * CPB; e += ST) {
        const int row = e % m, gg = e / m, j = j0 + gg;
        T val = T(0);
        if (j < r) {
          const double bv = sl.B[nd.row0 + row + (int64_t)j * sl.ldb];
          val = sl.colinv ? (T)(bv * sl.colinv[j]) : (T)bv;
        }
        sb[row + gg * LDS] = val;
      }
    } else {
      // children's u for this chunk (kv1 x ncol, kv2 x ncol), then
      // b = [b1; b2] - [T12 u2; T21 u1] (src/ulvfactor.jl:74)
      const T* u1g = ws + c1->wu + (int64_t)j0 * ld;
      const T* u2g = ws + c2->wu + (int64_t)j0 * ld;
      const T* u1p = u1g;  int64_t ldu1 = ld;
      const T* u2p = u2g;  int64_t ldu2 = ld;
      if (staged) {
        for (int e = tid; e < kv1 * ncol; e += ST) cpa(su1 + e, u1g + (e % kv1) + (int64_t)(e / kv1) * ld);
        for (int e = tid; e < kv2 * ncol; e += ST) cpa(su2 + e, u2g + (e % kv2) + (int64_t)(e / kv2) * ld);
        u1p = su1; ldu1 = kv1;
        u2p = su2; ldu2 = kv2;
        cpa_wait();
        __syncthreads();
      }
      for (int e = tid; e < m * CPB; e += ST) {
        const int row = e % m, gg = e / m;
        T val = T(0);
        if (gg < ncol) {
          const int64_t j = j0 + gg;
          T acc0 = T(0), acc1 = T(0);
          if (row < mr1) {
            val = ws[c1->wb + c1->mk + row + j * ld];
            const T* uu = u2p + (int64_t)gg * ldu2;
            int l = 0;
            for (; l + 1 < kv2; l += 2) {
              acc0 += T12p[row + l * mr1] * uu[l];
              acc1 += T12p[row + (l + 1) * mr1] * uu[l + 1];
            }
            if (l < kv2) acc0 += T12p[row + l * mr1] * uu[l];
          } else {
            const int i2 = row - mr1;
            val = ws[c2->wb + c2->mk + i2 + j * ld];
            const T* uu = u1p + (int64_t)gg * ldu1;
            int l = 0;
            for (; l + 1 < kv1; l += 2) {
              acc0 += T21p[i2 + l * mr2] * uu[l];
              acc1 += T21p[i2 + (l + 1) * mr2] * uu[l + 1];
            }
            if (l < kv1) acc0 += T21p[i2 + l * mr2] * uu[l];
          }
          val -= acc0 + acc1;
        }
        sb[row + gg * LDS] = val;
      }
      if (!nd.root) {
        // u accumulates W1^T u1 + W2^T u2 (src/ulvfactor.jl:89)
        for (int e = tid; e < kv * ncol; e += ST) {
          const int c = e % kv, gg = e / kv;
          const T* a1 = u1p + (int64_t)gg * ldu1;
          const T* a2 = u2p + (int64_t)gg * ldu2;
          T s = T(0);
          if (staged) {
            T s1 = T(0);
            for (int l = 0; l < kv1; ++l) s += sW1[l + c * ldW1] * a1[l];
            for (int l = 0; l < kv2; ++l) s1 += sW2[l + c * ldW2] * a2[l];
            s += s1;
          } else {
            for (int l = 0; l < kv1; ++l) s += (T)nd.W1[l + (int64_t)c * kv1] * a1[l];
            for (int l = 0; l < kv2; ++l) s += (T)nd.W2[l + (int64_t)c * kv2] * a2[l];
          }
          u[c + (int64_t)(j0 + gg) * ld] = s;
        }
      }
    }
    cpa_wait();   // leaves: the staged factor blocks
    __syncthreads();
    const int j = j0 + g;
    if (nd.root) {
      const T* A = Lp;
      const int32_t* piv = (const int32_t*)(fb + nd.fpiv);
      if (gl == 0) {
        T* col = sb + g * LDS;
        for (int c = 0; c < m; ++c) {
          const int p = piv[c];
          if (p != c) { const T t = col[c]; col[c] = col[p]; col[p] = t; }
        }
      }
      __syncwarp();
      T b[RPT];
#pragma unroll
      for (int s = 0; s < RPT; ++s) {
        const int row = gl + s * TPC;
        b[s] = row < m ? sb[row + g * LDS] : T(0);
      }
      lower_solve<T, TPC, RPT, true>(b, A, ldL, m, gl, s_rd);
      upper_solve<T, TPC, RPT>(b, A, ldL, m, gl, s_rd);
      if (__any_sync(0xffffffffu, j < r && failed<T, TPC>(b, A, ldL, m, gl))) {
        T* col = sb + g * LDS;
        lower_slow<T, TPC>(col, A, ldL, m, gl, true);
        upper_slow<T, TPC>(col, A, ldL, m, gl);
#pragma unroll
        for (int s = 0; s < RPT; ++s) {
          const int row = gl + s * TPC;
          b[s] = row < m ? col[row] : T(0);
        }
      }
      if (j < r) {
        T* x = ws + nd.wx + (int64_t)j * ld;
#pragma unroll
        for (int s = 0; s < RPT; ++s) {
          const int row = gl + s * TPC;
          if (row < m) x[row] = b[s];
        }
      }
      __syncthreads();
      continue;
    }
    if (mk > 0) {
      const T* tq = fb + nd.ftq;
      T b[RPT];
#pragma unroll
      for (int s = 0; s < RPT; ++s) {
        const int row = gl + s * TPC;
        b[s] = row < m ? sb[row + g * LDS] : T(0);
      }
      // b <- Q_ql^T b (src/ulvfactor.jl:42), reflectors in generation order
      for (int c = k - 1; c >= 0; --c) {
        const T tau = tq[c];   // 0: the reflector leaves b as it is
        const int p = mk + c;
        const T* v = Up + (int64_t)c * ldU;
        T d0 = T(0), d1 = T(0);
#pragma unroll
        for (int s = 0; s < RPT; ++s) {
          const int row = gl + s * TPC;
          const T vr = row < p ? v[row] : (row == p ? T(1) : T(0));
          if (s & 1) d1 += vr * b[s];
          else d0 += vr * b[s];
        }
        const T dot = gsum<TPC>(d0 + d1) * tau;
#pragma unroll
        for (int s = 0; s < RPT; ++s) {
          const int row = gl + s * TPC;
          const T vr = row < p ? v[row] : (row == p ? T(1) : T(0));
          b[s] -= dot * vr;
        }
      }
      // zloc = L1 \ b[0:mk] (trsm, src/ulvfactor.jl:48)
      lower_solve<T, TPC, RPT, false>(b, Lp, ldL, mk, gl, s_rd);
      if (__any_sync(0xffffffffu, j < r && failed<T, TPC>(b, Lp, ldL, mk, gl))) {
        reflect_slow<T, TPC>(sb + g * LDS, Up, ldU, tq, m, k, mk, gl);
        lower_slow<T, TPC>(sb + g * LDS, Lp, ldL, mk, gl, false);
      } else {
#pragma unroll
        for (int s = 0; s < RPT; ++s) {
          const int row = gl + s * TPC;
          if (row < m) sb[row + g * LDS] = b[s];
        }
      }
    }
    __syncthreads();
    // ---- outputs: b_red (:49), u (:51, :89), x[0:mk] = zloc (:65)
    for (int e = tid; e < (m - mk) * ncol; e += ST) {
      const int i = e % (m - mk), gg = e / (m - mk);
      const T* bb = sb + gg * LDS;
      T s0 = bb[mk + i], s1 = T(0);
      int l = 0;
      for (; l + 1 < nk; l += 2) {
        s0 -= L2p[i + l * ldL2] * bb[l];
        s1 -= L2p[i + (l + 1) * ldL2] * bb[l + 1];
      }
      if (l < nk) s0 -= L2p[i + l * ldL2] * bb[l];
      ws[nd.wb + mk + i + (int64_t)(j0 + gg) * ld] = s0 + s1;
    }
    for (int e = tid; e < kv * ncol; e += ST) {
      const int c = e % kv, gg = e / kv;
      const T* bb = sb + gg * LDS;
      T s0 = nd.leaf ? T(0) : u[c + (int64_t)(j0 + gg) * ld], s1 = T(0);
      int l = 0;
      for (; l + 1 < nk; l += 2) {
        s0 += Vap[l + c * ldVa] * bb[l];
        s1 += Vap[l + 1 + c * ldVa] * bb[l + 1];
      }
      if (l < nk) s0 += Vap[l + c * ldVa] * bb[l];
      u[c + (int64_t)(j0 + gg) * ld] = s0 + s1;
    }
    for (int e = tid; e < mk * ncol; e += ST) {
      const int i = e % mk, gg = e / mk;
      ws[nd.wx + i + (int64_t)(j0 + gg) * ld] = sb[i + gg * LDS];
    }
    __syncthreads();
  }
}

template <typename T, int TPC, int MR>
__global__ void __launch_bounds__(ST) ulv_solve_down_reg(const Task* __restrict__ tasks,
                                                         const Slot* __restrict__ slots, int stage_cap,
                                                         int nchunk) {
  constexpr int RPT = MR / TPC;
  constexpr int CPB = ST / TPC;
  extern __shared__ __align__(16) unsigned char smraw[];
  T* sQ = (T*)smraw;
  const Task tk = tasks[blockIdx.x / nchunk];
  const int jchunk = (blockIdx.x % nchunk) * CPB;
  const Node* nodes = tk.nodes;
  const Node& nd = nodes[tk.node];
  const Slot& sl = slots[tk.slot];
  T* ws = (T*)sl.ws;
  const int64_t ld = sl.ldws;
  const T* fb = (const T*)sl.fbase;
  const int n = nd.n, r = sl.r;
  pdl_trigger();
  if (jchunk >= r) {
    pdl_wait();
    return;
  }
  const int tid = threadIdx.x, g = tid / TPC, gl = tid % TPC;
  const T* x = ws + nd.wx;
  const T* Qt = fb + nd.fQt;
  if (!nd.root && nd.mk > 0 && n * nd.mk <= stage_cap) {
    for (int e = tid; e < n * nd.mk; e += ST) cpa(sQ + e, Qt + e);
    Qt = sQ;
    cpa_wait();
    __syncthreads();
  }
  pdl_wait();   // what follows reads the level before
  for (int j0 = jchunk; j0 < jchunk + CPB && j0 < r; j0 += CPB) {
    const int j = j0 + g;
    const bool act = j < r;
    T b[RPT];
#pragma unroll
    for (int s = 0; s < RPT; ++s) {
      const int row = gl + s * TPC;
      b[s] = (act && row < n) ? x[row + (int64_t)j * ld] : T(0);
    }
    if (!nd.root && nd.mk > 0) {
      // z[cols] = Q_lq^T z[cols]: reflectors i = mk-1 .. 0 (src/ulvfactor.jl:102)
      const T* tl = fb + nd.ftl;
      const int nl = min(nd.mk, n);
      for (int i = nl - 1; i >= 0; --i) {
        const T tau = tl[i];   // 0: the reflector leaves b as it is
        const T* v = Qt + (int64_t)i * n;
        T d0 = T(0), d1 = T(0);
#pragma unroll
        for (int s = 0; s < RPT; s += 2) {
          const int row = gl + s * TPC;
          if (row < n) d0 += v[row] * b[s];
          if (s + 1 < RPT && row + TPC < n) d1 += v[row + TPC] * b[s + 1];
        }
        const T w = gsum<TPC>(d0 + d1) * tau;
#pragma unroll
        for (int s = 0; s < RPT; ++s) {
          const int row = gl + s * TPC;
          if (row >= i && row < n) b[s] -= w * v[row];
        }
      }
    }
    if (!act) continue;
    if (nd.leaf) {
      const double sc = sl.colscale ? sl.colscale[j] : 1.0;
      double* out = sl.C + nd.col0 + (int64_t)j * sl.ldc;
#pragma unroll
      for (int s = 0; s < RPT; ++s) {
        const int row = gl + s * TPC;
        if (row < n) {
          const double v = sc * (double)b[s];
          if (sl.mode) out[row] += v;
          else out[row] = v;
        }
      }
    } else {
      const Node& c1 = nodes[nd.left];
      const Node& c2 = nodes[nd.right];
#pragma unroll
      for (int s = 0; s < RPT; ++s) {
        const int row = gl + s * TPC;
        if (row < n) {
          if (row < c1.nr) ws[c1.wx + c1.nk + row + (int64_t)j * ld] = b[s];
          else ws[c2.wx + c2.nk + (row - c1.nr) + (int64_t)j * ld] = b[s];
        }
      }
    }
  }
}

constexpr size_t kSolveSmemCap = 200 * 1024;

// A launch of ST threads per block, as a programmatic dependent of the one before
// it on the stream where pdl is set.
template <typename K, typename... A>
void launch_st(K kernel, int64_t blocks, size_t smem, cudaStream_t st, bool pdl, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3(ST);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = pdl ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <typename T, int TPC, int MR>
void up_launch(const Task* t, int64_t nt, const Slot* s, size_t want, int rmax, cudaStream_t st, bool pdl) {
  const size_t base = (size_t)(MR + 1) * (ST / TPC) * sizeof(T);
  size_t smem = base + want * sizeof(T);
  if (smem > kSolveSmemCap) smem = base;   // operands stay in global memory
  static SmemOptIn opt_in;
  opt_in((const void*)ulv_solve_up_reg<T, TPC, MR>, kSolveSmemCap);
  const int nchunk = (rmax + ST / TPC - 1) / (ST / TPC);
  launch_st(ulv_solve_up_reg<T, TPC, MR>, nt * nchunk, smem, st, pdl, t, s, (int64_t)((smem - base) / sizeof(T)), nchunk);
}

template <typename T, int TPC, int MR>
void down_launch(const Task* t, int64_t nt, const Slot* s, size_t want, int rmax, cudaStream_t st, bool pdl) {
  size_t smem = want * sizeof(T);
  if (smem > kSolveSmemCap) smem = 0;
  static SmemOptIn opt_in;
  opt_in((const void*)ulv_solve_down_reg<T, TPC, MR>, kSolveSmemCap);
  const int nchunk = (rmax + ST / TPC - 1) / (ST / TPC);
  launch_st(ulv_solve_down_reg<T, TPC, MR>, nt * nchunk, smem, st, pdl, t, s, (int)(smem / sizeof(T)), nchunk);
}

// 8 lanes per right-hand side: FP64 lists longer than two rounds of the SMs with
// at least 16 right-hand sides (32 to a block).
template <typename T>
bool narrow_groups(int64_t nt, int r, int sms) {
  return sizeof(T) == 8 && r >= 16 && nt * ((r + 7) / 8) > 2 * sms;
}

}  // namespace

bool solve_reg_fits(int mmax, int nmax) { return mmax <= 256 && nmax <= 256; }

int64_t solve_up_stage_need(int m, int k, int mk, int nk, int kv, bool leaf, bool root, int mr1, int mr2, int kv1,
                            int kv2) {
  return solve_up_stage_elems(m, k, mk, nk, kv, leaf, root, mr1, mr2, kv1, kv2, ST / 32);
}

// One warp (or a quarter of one) per right-hand-side column; the grid covers
// (node, column chunk) pairs so that few-node levels still fill SMs.
template <typename T>
void launch_ulv_solve_up_reg(const Task* t, int64_t nt, const Slot* s, int mmax, int64_t stage, int kvs, int r, int sms,
                             cudaStream_t st, bool pdl) {
  if (nt <= 0 || r <= 0) return;
  const size_t want = (size_t)stage;
  if constexpr (sizeof(T) == 8) {
    if (narrow_groups<T>(nt, r, sms) && mmax <= 128) {
      const size_t more = want + (size_t)kvs * (ST / 8 - ST / 32);   // the children's u of 32 columns
      if (mmax <= 64) up_launch<T, 8, 64>(t, nt, s, more, r, st, pdl);
      else up_launch<T, 8, 128>(t, nt, s, more, r, st, pdl);
      return;
    }
  }
  if (mmax <= 64) up_launch<T, 32, 64>(t, nt, s, want, r, st, pdl);
  else if (mmax <= 128) up_launch<T, 32, 128>(t, nt, s, want, r, st, pdl);
  else up_launch<T, 32, 256>(t, nt, s, want, r, st, pdl);
}

template <typename T>
void launch_ulv_solve_down_reg(const Task* t, int64_t nt, const Slot* s, int nmax, int mkmax, int r, int sms,
                               cudaStream_t st, bool pdl) {
  if (nt <= 0 || r <= 0) return;
  const size_t want = (size_t)nmax * mkmax;
  if constexpr (sizeof(T) == 8) {
    if (narrow_groups<T>(nt, r, sms) && nmax <= 128) {
      if (nmax <= 64) down_launch<T, 8, 64>(t, nt, s, want, r, st, pdl);
      else down_launch<T, 8, 128>(t, nt, s, want, r, st, pdl);
      return;
    }
  }
  if (nmax <= 64) down_launch<T, 32, 64>(t, nt, s, want, r, st, pdl);
  else if (nmax <= 128) down_launch<T, 32, 128>(t, nt, s, want, r, st, pdl);
  else down_launch<T, 32, 256>(t, nt, s, want, r, st, pdl);
}

template void launch_ulv_solve_up_reg<double>(const Task*, int64_t, const Slot*, int, int64_t, int, int, int, cudaStream_t,
                                              bool);
template void launch_ulv_solve_up_reg<float>(const Task*, int64_t, const Slot*, int, int64_t, int, int, int, cudaStream_t,
                                             bool);
template void launch_ulv_solve_down_reg<double>(const Task*, int64_t, const Slot*, int, int, int, int, cudaStream_t, bool);
template void launch_ulv_solve_down_reg<float>(const Task*, int64_t, const Slot*, int, int, int, int, cudaStream_t, bool);

}  // namespace hss
