// Persistent HSS x dense product: the whole product C = alpha A B + beta Y of
// a forest in one cooperative launch (reference src/matmul.jl:18-62).
//
// The level-by-level product needs 2 + (levels up) + (levels down) dependent
// launches, and the upper levels hold a few KB of work each, so their cost is
// launch and load latency.  Here every block of the grid is resident
// (cooperative launch) and the tree's dependencies are resolved on the device:
//
//   1. upsweep by climbing: for each (leaf, column chunk) pair a block forms
//      Z = V^T B (matmul.jl:34) and arrives at the parent's counter of that chunk.  The second
//      child to arrive computes the parent, Z = W1^T Z1 + W2^T Z2 (:39), and
//      climbs on; no block waits.  The B-terms of a branch's children, G1 = B12 Z2
//      and G2 = B21 Z1 (:51, :55), are a separate queue task, off the climb's
//      critical path.  The block that reaches a root forms the root's B-terms
//      and starts the downsweep of that tree (F of the root's children = G).
//   2. the leaf products D B (:46) are bulk units; upsweep and bulk units are
//      taken, upsweep first, from one global counter whenever no tree task is ready;
//   3. downsweep tasks go through a ready queue: the task of an internal node p,
//      enqueued once F_p is final and the B-terms of p's children are done, forms
//      F_c = G_c + R_c F_p (:50-56) for both children; the final task of a leaf
//      (C += U F, :47) is enqueued once F of the leaf is final and the leaf's bulk
//      unit is done.  Each pair of prerequisites meets on a per-node counter.
// A block claims a queue entry by taking a ticket (one atomicAdd, never
// retried) whenever produced entries are unclaimed, and then polls only its
// own entry's tag; between bulk units it looks for unclaimed entries first, so
// the tree's dependency chain runs underneath the bandwidth-bound bulk work.
// Once the bulk units are gone every block takes a ticket or leaves.  Waits
// are bounded: a block whose entry does not appear within the poll limit
// records DEV_TIMEOUT and exits.  The last block to finish resets the launch
// counters; the per-node counters are even between launches (each launch adds
// an even number), so consecutive launches need no clearing.  Small products (upsweep, translators, downsweep)
// are split over all warps of the block, because GB300's FP64 units issue a
// warp instruction only every 64 cycles per SM sub-partition.
//
// Two arithmetics share the code: FP64 (the product of hss_matmul) and
// double-float pairs on the FP32 pipe (the refinement residual, with the
// generators pre-split into pairs and B split on the fly).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "hss_df.cuh"
#include "hss_internal.h"
#include "hss_launch.h"

namespace hss {

namespace {

constexpr int PT = 256;                      // threads per block
constexpr int RC = 8;                        // widest column chunk
constexpr int kSyncChunks = 64;              // column chunks per node in the counter array
constexpr int LCH = 64;                      // rows of V staged per pass (leaf upsweep)
constexpr uint32_t kIdleLimit = 1u << 22;    // default polls of an idle block before it gives up
uint32_t g_idle_limit = kIdleLimit;          // host copy, passed to every launch (hss_set_option)
constexpr int PART_ELEMS = PT * 4;           // split-K partials (8-byte accumulators)

// launch counters, one 128-byte line each (the flat product uses the same
// words for its own)
enum { ST_HEAD = 0, ST_TAIL = 32, ST_BULK = 64, ST_DONE = 96, ST_WORDS = 128 };

// A queue entry is one 64-bit word, so that a consumer reads the task and its
// tag in one load: epoch (21 bits) | kind (1) | slot (16) | node (20) | column
// chunk (6).  Kinds: the node's downsweep task (a leaf's final task), or the
// B-terms of the node's children.
constexpr int QE_EPOCH = 43, QE_KIND = 42, QE_SLOT = 26, QE_NODE = 6;
enum { TK_DOWN = 0, TK_BTERM = 1 };

struct PmvArgs {
  const Task* leaves;
  const Slot* slots;
  uint32_t* state;       // launch counters
  unsigned long long* qent;   // queue entries
  const char* pf;        // translator generators, prefetched into L2 at the start
  int64_t pf_bytes;
  int32_t nleaves, ntasks, nchunk, nbulk;
  int32_t cw;            // columns per chunk (<= RC)
  uint32_t epoch;
  uint32_t idle_limit;   // polls of an idle block before DEV_TIMEOUT
};

// ---- arithmetic policies ----------------------------------------------------

struct PF64 {
  using E = double;
  struct Acc { double s; };
  __device__ static __forceinline__ Acc zero() { return Acc{0.0}; }
  __device__ static __forceinline__ void fma(Acc& a, E g, E x) { a.s = ::fma(g, x, a.s); }
  __device__ static __forceinline__ void acc(Acc& a, const Acc& b) { a.s += b.s; }
  __device__ static __forceinline__ void addE(Acc& a, E x) { a.s += x; }
  __device__ static __forceinline__ E fin(const Acc& a) { return a.s; }
  __device__ static __forceinline__ double dbl(const Acc& a) { return a.s; }
  __device__ static __forceinline__ const E* gen(const Slot&, const double* p) { return p; }
  __device__ static __forceinline__ E* ws(const Slot& s) { return (E*)s.ws; }
  __device__ static __forceinline__ E xin(double x) { return x; }
};

struct PDF {
  using E = float2;
  struct Acc { float h, l; };
  __device__ static __forceinline__ Acc zero() { return Acc{0.f, 0.f}; }
  __device__ static __forceinline__ void fma(Acc& a, E g, E x) { df_fma(a.h, a.l, g, x); }
  __device__ static __forceinline__ void acc(Acc& a, const Acc& b) { df_add(a.h, a.l, b.h, b.l); }
  __device__ static __forceinline__ void addE(Acc& a, E x) { df_add(a.h, a.l, x.x, x.y); }
  __device__ static __forceinline__ E fin(const Acc& a) { return df_norm(a.h, a.l); }
  __device__ static __forceinline__ double dbl(const Acc& a) { return (double)a.h + (double)a.l; }
  __device__ static __forceinline__ const E* gen(const Slot& s, const double* p) { return s.gdf + (p - s.gbase); }
  __device__ static __forceinline__ E* ws(const Slot& s) { return s.ws2; }
  __device__ static __forceinline__ E xin(double x) { return split_bits(x); }
};

// ---- device-side scheduling -------------------------------------------------

__device__ __forceinline__ uint32_t ld_vol(const uint32_t* p) { return *(const volatile uint32_t*)p; }

__device__ __forceinline__ void set_err(const Slot& sl, int code) {
  if (sl.err) atomicCAS((int*)sl.err, DEV_OK, code);
}

// counter of (node, chunk)
__device__ __forceinline__ int32_t* counter(const Slot& sl, int node, int ch) {
  return sl.sync + (int64_t)node * kSyncChunks + ch;
}

__device__ __forceinline__ unsigned long long qentry(uint32_t epoch, int kind, int slot, int node, int ch) {
  return ((unsigned long long)epoch << QE_EPOCH) | ((unsigned long long)kind << QE_KIND) |
         ((unsigned long long)slot << QE_SLOT) | ((unsigned long long)node << QE_NODE) | (unsigned long long)ch;
}

// Appends np <= 2 tasks (kind[i], slot, node[i], chunk) to the ready queue: one
// thread, after a barrier of the block and a fence that published the tasks' data.
__device__ void push(const PmvArgs& a, int slot, const int* node, const int* kind, int np, int ch, const Slot& sl) {
  if (np == 0) return;
  const uint32_t idx = atomicAdd(&a.state[ST_TAIL], (uint32_t)np);
  for (int i = 0; i < np; ++i) {
    if (idx + i >= (uint32_t)a.ntasks) {   // more tasks than the host counted: the tree tables disagree
      set_err(sl, DEV_BAD);
      return;
    }
    *(volatile unsigned long long*)&a.qent[idx + i] = qentry(a.epoch, kind[i], slot, node[i], ch);
  }
}

// Every non-root node's downsweep task (a leaf: its final task) has two
// prerequisites: its F is final, and either the B-terms of its children
// (branch) or its bulk unit (leaf) are done.  The second of the two events on
// the node's counter enqueues the task.  Counters are never reset: a launch
// adds an even number to each (a branch: two arrivals, then two events; a
// leaf: two events), so the second event of a pair is the one that reads an
// odd value.
__device__ void node_event(const PmvArgs& a, int slot, const Slot& sl, int node, int ch) {
  int32_t* c = counter(sl, node, ch);
  if (atomicAdd(c, 1) & 1) {
    // the first event's writes, observed through the counter, are published
    // with the entry (fence between observing and enqueueing)
    __threadfence();
    const int k = TK_DOWN;
    push(a, slot, &node, &k, 1, ch, sl);
  }
}

// F of both children of p (chunk ch) is final (thread 0, after the block's
// barrier and a fence): both counter updates are in flight together and the
// queue slots are taken with one atomic.
__device__ void release_children(const PmvArgs& a, int slot, const Slot& sl, const Node& p, int ch) {
  const int cs[2] = {p.left, p.right};
  int old[2];
  for (int i = 0; i < 2; ++i) old[i] = atomicAdd(counter(sl, cs[i], ch), 1);
  int go[2], kd[2] = {TK_DOWN, TK_DOWN}, np = 0;
  for (int i = 0; i < 2; ++i)
    if (old[i] & 1) go[np++] = cs[i];
  if (np == 0) return;
  __threadfence();   // as in node_event: the other events' writes go out with the entries
  push(a, slot, go, kd, np, ch, sl);
}

// ---- staging into shared memory ---------------------------------------------

// Asynchronous 8-byte copies global -> shared (cp.async), all of a phase in
// flight at once.  Only for data that no block writes during the launch (the
// generators): the copies go through L1.
__device__ __forceinline__ void cp8(void* s, const void* g) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(s)), "l"(g)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// rows x cols column-major block (global ld ldg) into shared memory (ld lds):
// warps take columns, lanes rows.
template <class E>
__device__ __forceinline__ void stage_gen(E* s, int lds, const E* g, int64_t ldg, int rows, int cols) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int c = w; c < cols; c += PT / 32)
    for (int l = lane; l < rows; l += 32) cp8(s + l + c * lds, g + l + (int64_t)c * ldg);
}

// The same for workspace blocks written by other blocks of this launch: loads
// that bypass L1 (an SM may hold a stale line of a neighbouring block).
template <class E>
__device__ __forceinline__ void stage_ws(E* s, int lds, const E* g, int64_t ldg, int rows, int cols) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int c = w; c < cols; c += PT / 32)
    for (int l = lane; l < rows; l += 32) s[l + c * lds] = __ldcg(g + l + (int64_t)c * ldg);
}

// ---- per-node work (one column chunk: columns j0 .. j0 + nc - 1) -------------

// Split-K layout of a small product over the block: op output slots (a power
// of two >= min(nout, PT)) x G = PT / op groups of terms.
__device__ __forceinline__ int out_slots(int nout) {
  int op = 1;
  while (op < nout && op < PT) op <<= 1;
  return op;
}

// The terms of one output of a small product: at most two strided segments,
// sum_{l < k1} a1[l sa1] b1[l sb1] + sum_{l < k2} a2[l sa2] b2[l sb2].  The
// call sites form the segment pointers once per output, so the inner loops
// hold no index arithmetic.
template <class E>
struct Terms {
  const E* a1;
  const E* b1;
  int sa1, sb1, k1;
  const E* a2;
  const E* b2;
  int sa2, sb2, k2;
};

template <class E>
__device__ __forceinline__ Terms<E> terms1(const E* a, int sa, const E* b, int sb, int k) {
  return Terms<E>{a, b, sa, sb, k, nullptr, nullptr, 0, 0, 0};
}

// acc[0..3] += the segment's terms l = g, g + G, ...: four independent chains
template <class P>
__device__ __forceinline__ void seg_acc(typename P::Acc (&acc)[4], const typename P::E* a, int sa,
                                        const typename P::E* b, int sb, int k, int g, int G) {
  int l = g;
  for (; l + 3 * G < k; l += 4 * G) {
    P::fma(acc[0], a[l * sa], b[l * sb]);
    P::fma(acc[1], a[(l + G) * sa], b[(l + G) * sb]);
    P::fma(acc[2], a[(l + 2 * G) * sa], b[(l + 2 * G) * sb]);
    P::fma(acc[3], a[(l + 3 * G) * sa], b[(l + 3 * G) * sb]);
  }
  for (; l < k; l += G) P::fma(acc[0], a[l * sa], b[l * sb]);
}

// out(o) = the sum of terms(o) for o < nout with every thread taking part (at
// most gmax groups of terms per output); epi(o, sum) consumes each result.
// `part` holds PT accumulators.
template <class P, class Setup, class Epi>
__device__ void sdot(int nout, typename P::Acc* part, Setup terms, Epi epi, int gmax = PT) {
  using Acc = typename P::Acc;
  const int op = max(out_slots(nout), PT / gmax), G = PT / op;
  const int slot = threadIdx.x % op, g = threadIdx.x / op;
  for (int o0 = 0; o0 < nout; o0 += op) {
    const int o = o0 + slot;
    Acc acc = P::zero();
    if (o < nout) {
      const Terms<typename P::E> t = terms(o);
      Acc a4[4] = {P::zero(), P::zero(), P::zero(), P::zero()};
      if (t.k1 > 0) seg_acc<P>(a4, t.a1, t.sa1, t.b1, t.sb1, t.k1, g, G);
      if (t.k2 > 0) seg_acc<P>(a4, t.a2, t.sa2, t.b2, t.sb2, t.k2, g, G);
      P::acc(a4[0], a4[1]);
      P::acc(a4[2], a4[3]);
      P::acc(a4[0], a4[2]);
      acc = a4[0];
    }
    if (G > 1) {
      __syncthreads();
      part[threadIdx.x] = acc;
      __syncthreads();
      if (g == 0 && o < nout)
        for (int gg = 1; gg < G; ++gg) P::acc(acc, part[gg * op + slot]);
    }
    if (g == 0 && o < nout) epi(o, acc);
  }
}

// Z = V^T B for one leaf (matmul.jl:34).  B is staged, V in passes of LCH rows
// (ld LCH + 1) through two buffers, the next pass's copies in flight while one
// is used; thread (output slot, group) keeps its partial sums over the passes.
// zsm (nullable, at least kv x nc elements, may overlay the V buffers) also
// receives Z (ld kv).
template <class P>
__device__ void leaf_up(const Slot& sl, const Node& nd, int j0, int nc, typename P::Acc* part,
                        typename P::E* sm, typename P::E* zsm = nullptr) {
  using E = typename P::E;
  using Acc = typename P::Acc;
  const int n = nd.gn, kv = nd.kv;
  if (kv == 0 || nc <= 0) return;
  const E* V = P::gen(sl, nd.V);
  E* ws = P::ws(sl);
  E* Xs = sm;                                      // n x RC
  E* Vb[2] = {sm + n * RC, sm + n * RC + (LCH + 1) * kv};   // LCH x kv each, ld LCH + 1
  const int npass = (n + LCH - 1) / LCH;
  auto issue = [&](int ps) {
    const int l0 = ps * LCH;
    stage_gen(Vb[ps & 1], LCH + 1, V + l0, n, min(LCH, n - l0), kv);
    cp_commit();
  };
  issue(0);
  if (npass > 1) issue(1);
  const int nout = kv * nc, op = out_slots(nout), G = PT / op;
  const int slot = threadIdx.x % op, g = threadIdx.x / op;
  const double* X = sl.B + nd.col0 + (int64_t)j0 * sl.ldb;
  {
    // four loads of a lane in flight before their conversions
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int q = w; q < nc; q += PT / 32)
      for (int l0 = 0; l0 < n; l0 += 128) {
        double v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int l = l0 + lane + 32 * u;
          v[u] = l < n ? __ldg(X + l + (int64_t)q * sl.ldb) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int l = l0 + lane + 32 * u;
          if (l < n) Xs[l + q * n] = P::xin(v[u]);
        }
      }
  }
  // nout <= 512 = 2 PT outputs per thread slot; four accumulator chains each
  Acc acc4[2][4];
#pragma unroll
  for (int s = 0; s < 2; ++s)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc4[s][c] = P::zero();
  for (int ps = 0; ps < npass; ++ps) {
    const int l0 = ps * LCH, nl = min(LCH, n - l0);
    const E* Vs = Vb[ps & 1];
    if (ps + 1 < npass) cp_wait<1>();
    else cp_wait<0>();
    __syncthreads();
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int o = s * op + slot;
      if (o < nout) {
        const int c = o % kv, q = o / kv;
        seg_acc<P>(acc4[s], Vs + c * (LCH + 1), 1, Xs + l0 + q * n, 1, nl, g, G);
      }
    }
    if (ps + 2 < npass) {
      __syncthreads();   // every thread is done with this buffer
      issue(ps + 2);
    }
  }
  if (zsm != nullptr) __syncthreads();   // every thread is done with the V buffers
  Acc acc[2];
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    P::acc(acc4[s][0], acc4[s][1]);
    P::acc(acc4[s][2], acc4[s][3]);
    P::acc(acc4[s][0], acc4[s][2]);
    acc[s] = acc4[s][0];
  }
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const int o = s * op + slot;
    if (G > 1) {
      __syncthreads();
      part[threadIdx.x] = acc[s];
      __syncthreads();
      if (g == 0 && o < nout)
        for (int gg = 1; gg < G; ++gg) P::acc(acc[s], part[gg * op + slot]);
    }
    if (g == 0 && o < nout) {
      const E z = P::fin(acc[s]);
      ws[nd.wz + (o % kv) + (int64_t)(j0 + o / kv) * sl.ldws] = z;
      if (zsm != nullptr) zsm[o] = z;
    }
  }
}

// Climb step at a non-root branch p once both children's Z are final:
// Z_p = W1^T Z1 + W2^T Z2 (matmul.jl:39).  The children's sizes and offsets come
// from p's descriptor (here a copy in shared memory).
template <class P>
__device__ void z_node(const Slot& sl, const Node& p, int j0, int nc, typename P::Acc* part, typename P::E* sm) {
  using E = typename P::E;
  using Acc = typename P::Acc;
  const int v1 = p.ckv[0], v2 = p.ckv[1], kv = p.kv;
  if (nc <= 0 || kv == 0) return;
  E* ws = P::ws(sl);
  const int64_t ld = sl.ldws;
  // W1, W2 column-major with odd leading dimensions (lanes take columns in the product)
  const int ld1 = v1 | 1, ld2 = v2 | 1;
  E* Z1 = sm;
  E* Z2 = Z1 + v1 * RC;
  E* W1s = Z2 + v2 * RC;
  E* W2s = W1s + ld1 * kv;
  stage_gen(W1s, ld1, P::gen(sl, p.W1), v1, v1, kv);
  stage_gen(W2s, ld2, P::gen(sl, p.W2), v2, v2, kv);
  cp_commit();
  stage_ws(Z1, v1, ws + p.cwz[0] + (int64_t)j0 * ld, ld, v1, nc);
  stage_ws(Z2, v2, ws + p.cwz[1] + (int64_t)j0 * ld, ld, v2, nc);
  cp_wait<0>();
  __syncthreads();
  sdot<P>(kv * nc, part,
          [&](int o) {
            const int c = o % kv, q = o / kv;
            return Terms<E>{W1s + c * ld1, Z1 + q * v1, 1, 1, v1, W2s + c * ld2, Z2 + q * v2, 1, 1, v2};
          },
          [&](int o, const Acc& s) { ws[p.wz + (o % kv) + (int64_t)(j0 + o / kv) * ld] = P::fin(s); });
}

// B-terms of branch p's children, G1 = B12 Z2 and G2 = B21 Z1 (matmul.jl:51,
// :55), into the children's F slots.  Off the upsweep's critical path: a queue
// task (the root's inline, its children's downsweep waits for them).
template <class P>
__device__ void bterm_node(const Slot& sl, const Node& p, int j0, int nc, typename P::Acc* part,
                           typename P::E* sm) {
  using E = typename P::E;
  using Acc = typename P::Acc;
  if (nc <= 0) return;
  const int v1 = p.ckv[0], v2 = p.ckv[1], u1 = p.cku[0], u2 = p.cku[1];
  E* ws = P::ws(sl);
  const int64_t ld = sl.ldws;
  E* Z1 = sm;
  E* Z2 = Z1 + v1 * RC;
  E* B12 = Z2 + v2 * RC;
  E* B21 = B12 + u1 * v2;
  stage_gen(B12, u1, P::gen(sl, p.B12), u1, u1, v2);
  stage_gen(B21, u2, P::gen(sl, p.B21), u2, u2, v1);
  cp_commit();
  stage_ws(Z1, v1, ws + p.cwz[0] + (int64_t)j0 * ld, ld, v1, nc);
  stage_ws(Z2, v2, ws + p.cwz[1] + (int64_t)j0 * ld, ld, v2, nc);
  cp_wait<0>();
  __syncthreads();
  sdot<P>((u1 + u2) * nc, part,
          [&](int o) {
            if (o < u1 * nc) return terms1<E>(B12 + o % u1, u1, Z2 + (o / u1) * v2, 1, v2);
            const int o2 = o - u1 * nc;
            return terms1<E>(B21 + o2 % u2, u2, Z1 + (o2 / u2) * v1, 1, v1);
          },
          [&](int o, const Acc& s) {
            if (o < u1 * nc) ws[p.cwf[0] + (o % u1) + (int64_t)(j0 + o / u1) * ld] = P::fin(s);
            else ws[p.cwf[1] + ((o - u1 * nc) % u2) + (int64_t)(j0 + (o - u1 * nc) / u2) * ld] = P::fin(s);
          });
}

// Arrival of a finished node x (its Z of chunk ch written by this block) at its
// parent; the second child to arrive climbs.  While thread 0 fences and
// arrives, warp 1 enqueues the B-term task of x (a branch) and warp 2 copies
// the parent's descriptor into shared memory, so the next step reads no
// descriptor from global memory.  At the root the block forms the root's
// B-terms, which are F of the root's children, and releases them.
template <class P>
__device__ void climb_from(const PmvArgs& a, int slot, const Slot& sl, const Node* nodes, int node, int ch,
                           typename P::Acc* part, typename P::E* sm) {
  __shared__ int s_go;
  __shared__ Node s_node;
  const int j0 = ch * a.cw, nc = min(a.cw, sl.r - j0);
  const Node* x = &nodes[node];
  for (;;) {
    const int xpar = x->parent;
    const bool xroot = x->root != 0, xbranch = !x->leaf;
    __syncthreads();   // x's Z is written; nobody reads s_node any more
    if (xroot) return;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
      __threadfence();   // publishes the block's writes (cumulative over the barrier)
      const int old = atomicAdd(counter(sl, xpar, ch), 1);
      s_go = old & 1;
      if (old & 1) __threadfence();   // acquire: the sibling's Z is read after the barrier below
    } else if (threadIdx.x == 32 && xbranch) {
      __threadfence();
      const int k = TK_BTERM;
      push(a, slot, &node, &k, 1, ch, sl);
    } else if (w == 2) {
      const unsigned long long* src = (const unsigned long long*)&nodes[xpar];
      unsigned long long* dst = (unsigned long long*)&s_node;
      for (int i = lane; i < (int)(sizeof(Node) / 8); i += 32) dst[i] = src[i];
    }
    __syncthreads();
    if (!s_go) return;
    const Node& p = s_node;
    node = xpar;
    if (p.root) {
      bterm_node<P>(sl, p, j0, nc, part, sm);
      __syncthreads();
      if (threadIdx.x == 0) {
        __threadfence();
        release_children(a, slot, sl, p, ch);
      }
      return;
    }
    z_node<P>(sl, p, j0, nc, part, sm);
    x = &s_node;
  }
}

// Downsweep task of a non-root branch p (F_p final, its children's B-terms G_c
// done): F_c = G_c + R_c F_p for both children (matmul.jl:50-56), in place over G_c.
template <class P>
__device__ void down_node(const Slot& sl, const Node& p, int j0, int nc, typename P::Acc* part, typename P::E* sm) {
  using E = typename P::E;
  using Acc = typename P::Acc;
  if (nc <= 0) return;
  const int u1 = p.cku[0], u2 = p.cku[1], kp = p.ku;
  const int64_t f1 = p.cwf[0], f2 = p.cwf[1];
  E* ws = P::ws(sl);
  const int64_t ld = sl.ldws;
  E* Fp = sm;                 // kp x RC
  E* R1 = Fp + kp * RC;       // u1 x kp
  E* R2 = R1 + u1 * kp;       // u2 x kp
  E* G1 = R2 + u2 * kp;       // u1 x RC: the children's B-terms
  E* G2 = G1 + u1 * RC;       // u2 x RC
  stage_gen(R1, u1, P::gen(sl, p.R1), u1, u1, kp);
  stage_gen(R2, u2, P::gen(sl, p.R2), u2, u2, kp);
  cp_commit();
  stage_ws(Fp, kp, ws + p.wf + (int64_t)j0 * ld, ld, kp, nc);
  stage_ws(G1, u1, ws + f1 + (int64_t)j0 * ld, ld, u1, nc);
  stage_ws(G2, u2, ws + f2 + (int64_t)j0 * ld, ld, u2, nc);
  cp_wait<0>();
  __syncthreads();
  sdot<P>((u1 + u2) * nc, part,
          [&](int o) {
            if (o < u1 * nc) return terms1<E>(R1 + o % u1, u1, Fp + (o / u1) * kp, 1, kp);
            const int o2 = o - u1 * nc;
            return terms1<E>(R2 + o2 % u2, u2, Fp + (o2 / u2) * kp, 1, kp);
          },
          [&](int o, const Acc& s) {
            const bool first = o < u1 * nc;
            const int o2 = first ? o : o - u1 * nc;
            const int uc = first ? u1 : u2;
            Acc t = s;
            P::addE(t, (first ? G1 : G2)[o2]);   // G[i + q uc] with i = o2 % uc, q = o2 / uc
            ws[(first ? f1 : f2) + (o2 % uc) + (int64_t)(j0 + o2 / uc) * ld] = P::fin(t);
          });
}

// out(i, q) = sum_l A(i + l*lda) Xs(l + q*ldx) for i < m, q < NQ, l < K, A from
// global memory (read-only), Xs staged; `epi(i, q, acc)` consumes each result and
// returns the FP64 value written (for the column sums of squares when cn != 0).
// Threads: row slot ii of rp (a power of two >= rows of the pass), split-K group g.
template <class P, int NQ, class Epi>
__device__ void rows_cols(const typename P::E* __restrict__ A, int m, int K, int64_t lda,
                          const typename P::E* Xs, int ldx, typename P::Acc* part, double* cn, Epi epi) {
  using Acc = typename P::Acc;
  const int tid = threadIdx.x;
  double sq[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) sq[q] = 0.0;
  for (int r0 = 0; r0 < m; r0 += PT) {
    const int rows = min(PT, m - r0);
    int rp = 1;
    while (rp < rows) rp <<= 1;
    const int G = PT / rp;
    const int ii = tid % rp, g = tid / rp;
    const int i = r0 + ii;
    const bool act = ii < rows;
    Acc acc[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) acc[q] = P::zero();
    if (act) {
      const typename P::E* a = A + i;
#pragma unroll 8
      for (int l = g; l < K; l += G) {
        const typename P::E d = __ldg(a + (int64_t)l * lda);
#pragma unroll
        for (int q = 0; q < NQ; ++q) P::fma(acc[q], d, Xs[l + q * ldx]);
      }
    }
    if (G > 1) {
      __syncthreads();
#pragma unroll
      for (int q = 0; q < NQ; ++q) part[(g * rp + ii) * NQ + q] = acc[q];
      __syncthreads();
      if (g == 0 && act) {
        for (int gg = 1; gg < G; ++gg)
#pragma unroll
          for (int q = 0; q < NQ; ++q) P::acc(acc[q], part[(gg * rp + ii) * NQ + q]);
      }
    }
    if (g == 0 && act) {
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const double v = epi(i, q, acc[q]);
        sq[q] = fma(v, v, sq[q]);
      }
    }
  }
  if (cn != nullptr) {
    const int lane = tid & 31;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      double v = sq[q];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0 && v != 0.0) atomicAdd(cn + q, v);
    }
  }
}

// Runs rows_cols over nc <= RC columns in groups of 4, 2, 1; `epi(i, q, acc)`
// receives the absolute column q within the pass.
template <class P, class Epi>
__device__ void rows_cols_n(const typename P::E* A, int m, int K, int64_t lda, const typename P::E* Xs, int ldx,
                            int nc, typename P::Acc* part, double* cn, Epi epi) {
  int q0 = 0;
  auto run = [&](auto nq) {
    constexpr int NQ = decltype(nq)::value;
    rows_cols<P, NQ>(A, m, K, lda, Xs + q0 * ldx, ldx, part, cn ? cn + q0 : nullptr,
                     [&](int i, int q, const typename P::Acc& s) { return epi(i, q0 + q, s); });
    q0 += NQ;
  };
  while (nc - q0 >= 4) run(std::integral_constant<int, 4>());
  if (nc - q0 >= 2) run(std::integral_constant<int, 2>());
  if (nc - q0 >= 1) run(std::integral_constant<int, 1>());
}

// Bulk unit: the leaf product D B for one column chunk (matmul.jl:46).  FP64:
// C = alpha D B + beta Y; pairs: D B kept in the pair buffer for the final task.
// A single-leaf tree (the leaf is the root) finishes here, column norms included.
template <class P>
__device__ void bulk_unit(const PmvArgs& a, int u, typename P::Acc* part, typename P::E* sm) {
  using E = typename P::E;
  using Acc = typename P::Acc;
  const int t = u / a.nchunk, ch = u % a.nchunk;
  const Task tk = a.leaves[t];
  const Slot& sl = a.slots[tk.slot];
  const Node& nd = tk.nodes[tk.node];
  const int j0 = ch * a.cw;
  if (ch == 0 && !nd.root && nd.ku > 0) {
    // U is read by the leaf's final tasks at the end of the downsweep: into L2 now
    const char* ub = (const char*)P::gen(sl, nd.U);
    const int64_t bytes = (int64_t)nd.gm * nd.ku * (int64_t)sizeof(E);
    for (int64_t off = (int64_t)threadIdx.x * 128; off < bytes; off += PT * 128)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(ub + off));
  }
  if (j0 < sl.r) {
    const int nc = min(a.cw, sl.r - j0), m = nd.gm, n = nd.gn;
    E* Xs = sm;
    __syncthreads();
    const double* X = sl.B + nd.col0 + (int64_t)j0 * sl.ldb;
    for (int e = threadIdx.x; e < n * nc; e += PT) {
      const int l = e % n, q = e / n;
      Xs[l + q * n] = P::xin(__ldg(X + l + (int64_t)q * sl.ldb));
    }
    __syncthreads();
    const E* D = P::gen(sl, nd.D);
    double* C = sl.C + nd.row0 + (int64_t)j0 * sl.ldc;
    const double* Y = sl.Y ? sl.Y + nd.row0 + (int64_t)j0 * sl.ldy : nullptr;
    const bool yterm = sl.beta != 0.0 && Y != nullptr;
    double* cn = (nd.root && sl.colnorm2) ? sl.colnorm2 + j0 : nullptr;
    constexpr bool pairs = !std::is_same<E, double>::value;
    if (pairs && !nd.root) {
      E* T = (E*)sl.tmp + nd.row0 + (int64_t)j0 * sl.ldt2;
      rows_cols_n<P>(D, m, n, m, Xs, n, nc, part, nullptr, [&](int i, int q, const Acc& s) {
        T[i + (int64_t)q * sl.ldt2] = P::fin(s);
        return 0.0;
      });
    } else {
      rows_cols_n<P>(D, m, n, m, Xs, n, nc, part, cn, [&](int i, int q, const Acc& s) {
        double v = sl.alpha * P::dbl(s);
        if (yterm) v += sl.beta * __ldcg(Y + i + (int64_t)q * sl.ldy);
        C[i + (int64_t)q * sl.ldc] = v;
        return v;
      });
    }
  }
  if (!nd.root) {
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      node_event(a, tk.slot, sl, tk.node, ch);
    }
  }
}

// Final task of a non-root leaf chunk (F final, bulk done): C += alpha U F
// (matmul.jl:47), or for pairs C = alpha (D B + U F) + beta Y, with the column
// sums of squares.  Thread (row ii, group g) takes the columns of group g
// whole (no split over K, no cross-thread sums), FQ at a time, and loads
// its epilogue operands (D B, Y, or C) before the product, so that their
// latency overlaps the loop over U's columns.
template <class P>
__device__ void final_leaf(const Slot& sl, const Node& nd, int j0, int nc, typename P::Acc* part,
                           typename P::E* sm) {
  using E = typename P::E;
  using Acc = typename P::Acc;
  constexpr bool pairs = !std::is_same<E, double>::value;
  constexpr int FQ = 2;   // columns per pass (registers: the launch allows 64 per thread)
  (void)part;
  if (nc <= 0) return;
  const int m = nd.gm, ku = nd.ku;
  E* ws = P::ws(sl);
  E* Fs = sm;                              // ku x RC
  const E* U = P::gen(sl, nd.U);
  __syncthreads();
  stage_ws(Fs, ku, ws + nd.wf + (int64_t)j0 * sl.ldws, sl.ldws, ku, nc);
  __syncthreads();
  double* C = sl.C + nd.row0 + (int64_t)j0 * sl.ldc;
  double* cn = sl.colnorm2 ? sl.colnorm2 + j0 : nullptr;
  const E* T = pairs ? (const E*)sl.tmp + nd.row0 + (int64_t)j0 * sl.ldt2 : nullptr;
  const double* Y = sl.Y ? sl.Y + nd.row0 + (int64_t)j0 * sl.ldy : nullptr;
  const bool yterm = pairs && sl.beta != 0.0 && Y != nullptr;
  const int tid = threadIdx.x;
  for (int r0 = 0; r0 < m; r0 += PT) {
    const int rows = min(PT, m - r0);
    int rp = 1;
    while (rp < rows) rp <<= 1;
    const int G = PT / rp, ii = tid % rp, g = tid / rp;
    const int i = r0 + ii;
    const int cpg = (nc + G - 1) / G, q0 = g * cpg, q1 = min(nc, q0 + cpg);
    for (int qb = q0; qb < q1; qb += FQ) {
      const int nq = min(FQ, q1 - qb);
      const bool act = ii < rows;
      // epilogue operands first
      E tv[FQ];
      double yv[FQ];
#pragma unroll
      for (int q = 0; q < FQ; ++q) {
        tv[q] = E{};
        yv[q] = 0.0;
        if (act && q < nq) {
          if (pairs) {
            tv[q] = __ldcg(T + i + (int64_t)(qb + q) * sl.ldt2);
            if (yterm) yv[q] = __ldcg(Y + i + (int64_t)(qb + q) * sl.ldy);
          } else {
            yv[q] = __ldcg(C + i + (int64_t)(qb + q) * sl.ldc);
          }
        }
      }
      Acc acc[FQ];
#pragma unroll
      for (int q = 0; q < FQ; ++q) acc[q] = P::zero();
      if (act) {
        const E* a = U + i;
#pragma unroll 8
        for (int l = 0; l < ku; ++l) {
          const E d = __ldg(a + (int64_t)l * m);
#pragma unroll
          for (int q = 0; q < FQ; ++q)
            if (q < nq) P::fma(acc[q], d, Fs[l + (qb + q) * ku]);
        }
      }
#pragma unroll
      for (int q = 0; q < FQ; ++q) {
        double v = 0.0;
        if (act && q < nq) {
          if (pairs) {
            Acc t = acc[q];
            P::addE(t, tv[q]);
            v = sl.alpha * P::dbl(t);
            if (yterm) v += sl.beta * yv[q];
          } else {
            v = yv[q] + sl.alpha * P::dbl(acc[q]);
          }
          C[i + (int64_t)(qb + q) * sl.ldc] = v;
        }
        if (cn != nullptr) {
          // a warp lies within one group when rp >= 32: warp sums, one atomic per column
          double v2 = v * v;
          if (rp >= 32) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v2 += __shfl_xor_sync(0xffffffffu, v2, o);
            if ((tid & 31) == 0 && q < nq && v2 != 0.0) atomicAdd(cn + qb + q, v2);
          } else if (q < nq && v2 != 0.0) {
            atomicAdd(cn + qb + q, v2);
          }
        }
      }
    }
  }
}

template <class P>
__global__ void __launch_bounds__(PT, 4) pmv_kernel(PmvArgs a) {
  using E = typename P::E;
  using Acc = typename P::Acc;
  extern __shared__ __align__(16) unsigned char pmv_smem[];
  Acc* part = (Acc*)pmv_smem;                    // PART_ELEMS split-K partials
  E* sm = (E*)pmv_smem + PART_ELEMS;             // per-phase staging
  __shared__ int s_cmd, s_x, s_y, s_k;

  // the translators are read by the tree chain: have them in L2 before it starts
  for (int64_t off = ((int64_t)blockIdx.x * PT + threadIdx.x) * 128; off < a.pf_bytes;
       off += (int64_t)gridDim.x * PT * 128)
    asm volatile("prefetch.global.L2::evict_last [%0];" ::"l"(a.pf + off));

  // Work units of one counter: the nbulk (leaf, chunk) upsweep units first (they
  // start the tree chain), then the nbulk bulk units; claimed queue entries first.
  const uint32_t nwork = 2u * (uint32_t)a.nbulk;
  uint32_t idle = 0;
  int ticket = -1;   // queue entry this block has claimed (thread 0)
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) {
      int cmd = 0;
      if (ticket < 0) {
        const uint32_t hd = ld_vol(&a.state[ST_HEAD]);
        if (hd < ld_vol(&a.state[ST_TAIL])) {          // produced, unclaimed entries
          const uint32_t t = atomicAdd(&a.state[ST_HEAD], 1u);
          if (t < (uint32_t)a.ntasks) ticket = (int)t;
        }
        if (ticket < 0) {
          if (ld_vol(&a.state[ST_BULK]) < nwork) {
            const uint32_t u = atomicAdd(&a.state[ST_BULK], 1u);
            if (u < nwork) {
              s_x = (int)u;
              cmd = 2;
            }
          }
          if (cmd == 0) {                                // no bulk left: claim or leave
            const uint32_t t = hd < (uint32_t)a.ntasks ? atomicAdd(&a.state[ST_HEAD], 1u) : (uint32_t)a.ntasks;
            if (t < (uint32_t)a.ntasks) ticket = (int)t;
            else cmd = 3;
          }
        }
      }
      if (ticket >= 0) {
        const unsigned long long w = *(const volatile unsigned long long*)&a.qent[ticket];
        if ((uint32_t)(w >> QE_EPOCH) == a.epoch) {
          __threadfence();   // acquire: the task's inputs are read after the barrier below
          s_x = (int)((w >> QE_SLOT) & 0xffffu);
          s_y = (int)(w & ((1u << QE_SLOT) - 1));   // node * kSyncChunks + chunk
          s_k = (int)((w >> QE_KIND) & 1u);
          cmd = 1;
          ticket = -1;
        }
      }
      if (cmd == 0) {
        if (++idle > a.idle_limit) {
          set_err(a.slots[0], DEV_TIMEOUT);
          cmd = 3;
        } else {
          __nanosleep(32);
        }
      } else {
        idle = 0;
      }
      s_cmd = cmd;
    }
    __syncthreads();
    const int cmd = s_cmd;
    if (cmd == 3) break;
    if (cmd == 1) {
      const int slot = s_x, node = s_y / kSyncChunks, ch = s_y % kSyncChunks;
      const Slot& sl = a.slots[slot];
      const Node* nodes = sl.nodes;
      const Node& x = nodes[node];
      const int j0 = ch * a.cw, nc = min(a.cw, sl.r - j0);
      if (s_k == TK_BTERM) {
        bterm_node<P>(sl, x, j0, nc, part, sm);
        __syncthreads();
        if (threadIdx.x == 0) {
          __threadfence();
          node_event(a, slot, sl, node, ch);
        }
      } else if (x.leaf) {
        final_leaf<P>(sl, x, j0, nc, part, sm);
      } else {
        down_node<P>(sl, x, j0, nc, part, sm);
        __syncthreads();
        if (threadIdx.x == 0) {
          __threadfence();
          release_children(a, slot, sl, x, ch);
        }
      }
    } else if (cmd == 2) {
      const int u = s_x;
      if (u < a.nbulk) {
        // upsweep unit (leaf, chunk): Z = V^T B, then climb
        const int ch = u % a.nchunk;
        const Task tk = a.leaves[u / a.nchunk];
        const Slot& sl = a.slots[tk.slot];
        const Node& nd = tk.nodes[tk.node];
        if (!nd.root) {
          const int j0 = ch * a.cw;
          leaf_up<P>(sl, nd, j0, min(a.cw, sl.r - j0), part, sm);
          climb_from<P>(a, tk.slot, sl, tk.nodes, tk.node, ch, part, sm);
        }
      } else {
        bulk_unit<P>(a, u - a.nbulk, part, sm);
      }
    }
  }

  // the last block out resets the launch counters
  if (threadIdx.x == 0) {
    __threadfence();
    const uint32_t d = atomicAdd(&a.state[ST_DONE], 1u);
    if (d == gridDim.x - 1) {
      a.state[ST_HEAD] = 0;
      a.state[ST_TAIL] = 0;
      a.state[ST_BULK] = 0;
      __threadfence();
      a.state[ST_DONE] = 0;
    }
  }
}

template <class P>
struct Occ {
  size_t smem = 0;
  int blocks = 0;
};

template <class P>
int resident_blocks(size_t smem, int device) {
  static Occ<P> cache[8];
  if (device < 0 || device >= 8) device = 0;
  Occ<P>& c = cache[device];
  if (c.smem == smem && c.blocks > 0) return c.blocks;
  if (smem > 48 * 1024) cudaFuncSetAttribute(pmv_kernel<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  int per_sm = 0, sms = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pmv_kernel<P>, PT, smem) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return 0;
  c.smem = smem;
  c.blocks = per_sm * sms;
  return c.blocks;
}

}  // namespace

// Shared memory (elements of 8 bytes) the persistent product needs for leaves
// of at most nleaf columns, ranks of at most kmax; mcap receives the part
// available for staged translators.
size_t pmv_smem_elems(int nleaf, int kmax, int* mcap) {
  const size_t k = kmax > 0 ? kmax : 1;
  const size_t up = (size_t)nleaf * RC + 2 * (size_t)(LCH + 1) * k;   // X + two V buffers
  const size_t bulk = (size_t)nleaf * RC;
  const size_t fin = k * RC;
  const size_t down = 3 * k * RC + 2 * k * k;                         // F_p, R1, R2, G1, G2
  const size_t climb = 2 * k * RC + 2 * (k | 1) * k;                  // Z1, Z2, W1, W2
  const size_t bterm = 2 * k * RC + 2 * k * k;                        // Z1, Z2, B12, B21
  const size_t total = PART_ELEMS + std::max(std::max(std::max(up, bulk), std::max(fin, down)), std::max(climb, bterm));
  if (mcap) *mcap = (int)(total - PART_ELEMS);
  return total;
}

bool pmv_fits(int nleaf, int mleaf, int kmax) {
  return nleaf <= 512 && mleaf <= 1 << 20 && kmax <= 64 && pmv_smem_elems(nleaf, kmax, nullptr) * 8 <= 160 * 1024;
}

int pmv_chunks(bool pairs, int rmax) {
  const int cw = pairs ? RC : 4;
  const int nc = std::max(1, (rmax + cw - 1) / cw);
  return nc <= kSyncChunks ? nc : 0;
}
int64_t pmv_queue_entries(int64_t ntasks, int64_t ninner, int chunks) { return (ntasks + ninner) * chunks; }
int64_t pmv_state_words() { return ST_WORDS; }
uint32_t pmv_epoch_limit() { return (1u << (64 - QE_EPOCH)) - 1; }
bool pmv_queue_fits(int64_t nodes, int64_t slots) {
  return nodes <= (int64_t(1) << (QE_SLOT - QE_NODE)) && slots <= (int64_t(1) << (QE_EPOCH - QE_SLOT));
}
int pmv_sync_chunks() { return kSyncChunks; }
void pmv_set_poll_limit(uint32_t polls) { g_idle_limit = polls == 0 ? kIdleLimit : polls; }
uint32_t pmv_poll_limit() { return g_idle_limit; }

cudaError_t launch_pmv(bool pairs, const Task* leaves, int64_t nleaves, const Slot* slots, int64_t ntasks,
                       int64_t ninner, int rmax,
                       int nleaf, int kmax, uint32_t* state, unsigned long long* qent, uint32_t epoch,
                       const void* prefetch,
                       int64_t prefetch_bytes, int device, cudaStream_t st) {
  if (nleaves <= 0) return cudaSuccess;
  const size_t smem = pmv_smem_elems(nleaf, kmax, nullptr) * 8;
  PmvArgs a;
  a.leaves = leaves;
  a.slots = slots;
  a.state = state;
  a.qent = qent;
  a.nleaves = (int32_t)nleaves;
  a.cw = pairs ? RC : 4;   // FP64: narrower chunks spread the slow FP64 work over more SMs
  a.nchunk = pmv_chunks(pairs, rmax);
  if (a.nchunk == 0) return cudaErrorInvalidValue;
  a.nbulk = (int32_t)(nleaves * a.nchunk);
  a.ntasks = (int32_t)pmv_queue_entries(ntasks, ninner, a.nchunk);
  a.epoch = epoch;
  a.pf = (const char*)prefetch;
  a.pf_bytes = prefetch ? prefetch_bytes : 0;
  a.idle_limit = g_idle_limit;
  void* args[] = {&a};
  const int cap = pairs ? resident_blocks<PDF>(smem, device) : resident_blocks<PF64>(smem, device);
  if (cap <= 0) return cudaErrorLaunchOutOfResources;
  // every block must be resident; more blocks than work units would only poll
  const unsigned grid = (unsigned)std::min<int64_t>(cap, std::max<int64_t>(1, 2 * (int64_t)a.nbulk));
  return pairs ? cudaLaunchCooperativeKernel((void*)pmv_kernel<PDF>, grid, PT, args, smem, st)
               : cudaLaunchCooperativeKernel((void*)pmv_kernel<PF64>, grid, PT, args, smem, st);
}

}  // namespace hss
