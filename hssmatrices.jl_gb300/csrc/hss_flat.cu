// Flat persistent HSS x dense product (FP64, few columns): C = alpha A B + beta Y
// of a forest in one cooperative launch (reference src/matmul.jl:18-62).
//
// With few columns the tree's chain of dependent small products and the FP64 pipe
// (a warp instruction every 64 clocks and quarter SM, active lanes or not) bound the
// product, not the generators' bytes.  The leaves are cut into groups, maximal
// subtrees (not whole trees) of at most 1, 2, 4 or 8 leaves, and one block takes a
// group and a chunk of columns through the tree:
//
//   A. per group, Z = V^T B of its leaves (matmul.jl:34), Z = W1^T Z1 + W2^T Z2 of
//      its branches (:39), the B-terms these feed (G_sibling = B Z, :51/:55), and
//      the group's contributions to the Z of the branches above it,
//      W_a^T ... W_x^T Z (the terms of :39 unrolled along the path);
//   B. per non-root branch above the groups, Z = the sum of its groups'
//      contributions (in leaf order, so that the result does not depend on the
//      schedule), then the B-term it feeds;
//   C. per group, F along the path from the root, F_c = G_c + R_c F_p (:50-56, F of
//      the root's children = G), then inside the group, then C += alpha U F (:47).
//
// A phase starts once every unit of the one before it has finished (a count of
// finished units).  The leaf products C = alpha D B + beta Y (:46), 32 rows a
// unit, have no tree dependency: four of a block's twenty warps do nothing else,
// the others join where they have no group or wait for a leaf's pieces.
//
// Why groups: a chain carried by every leaf costs 10 M of 26 M multiply-adds at
// n = 65536, k = 32 in repeated translators; with groups of four 0.9 M are left, and
// one block an SM keeps the chain's steps from queueing behind other blocks'
// products.  Why lanes: small products give every output eight or four lanes, which
// split the inner terms and add up by shuffles, so that a step has one barrier and no
// partial sums in shared memory; products with enough rows (B-terms, R inside the
// group, U F, D B) give a row a lane and add nothing up.  The teams of eight warps
// share a group's leaves; then one carries the chain while the other does the B-terms.
//
// Measured, us (each leaf its own chain, four blocks an SM -> groups): n = 65536, k =
// 32: r = 1 99 -> 68, 2 141 -> 113, 4 226 -> 208; n = 16384 r = 1 62 -> 40; n = 10007,
// leaves of 39 rows, k = 20: r = 1 60 -> 38, 7 (queued product) 129 -> 71; n = 512 r = 1
// 32 -> 23; the runs of rows32 add up to 4 % (n = 65536, r = 1).  Inside that launch (57): leaves 12, inner branches 4, chain
// 9, rest of phase A and the wait 4, phase B 6, path 8, inner 6, U F 6.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>

#include "hss_internal.h"
#include "hss_launch.h"
#include "hss_optin.h"

namespace hss {

namespace {

constexpr int TM = 256;              // threads of a team
constexpr int TT = 2 * TM;           // threads of the tree warps: two teams
constexpr int FT = TT + 128;         // and four warps of leaf products
constexpr int kFlatCw = 4;           // widest column chunk
constexpr int PR = 32;               // rows per leaf-product unit
constexpr int GN = 2 * kFlatGroup - 1;   // nodes of a group
enum { FL_AFIN = 0, FL_BFIN = 32, FL_D = 64, FL_DONE = 96 };   // launch counters, a 128-byte line each

struct FlatArgs {
  const Task* leaves;           // leaf list (a subtree's leaves are contiguous)
  const Node* nodes;
  const FlatLink* links;        // by node
  const FlatGroup* groups;      // in leaf order
  const FlatBranch* branches;   // non-root branches above the groups
  const Slot* slots;
  uint32_t* state;
  double* ctb;                  // contributions: ((depth * ngroup + group) * nchunk + chunk) * kk + (c + q km)
  uint32_t* dcnt;               // finished leaf-product pieces per (leaf, chunk); zero between launches
  int32_t nleaves, ngroup, nbranch, nchunk, npiece, dep, km, nbuf, nleaf;
  uint32_t idle_limit;          // polls of a waiting block before DEV_TIMEOUT
};

__device__ __forceinline__ uint32_t ld_acq(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t ld_vol(const uint32_t* p) { return *(const volatile uint32_t*)p; }

__device__ __forceinline__ void set_err(const Slot& sl, int code) {
  if (sl.err) atomicCAS((int*)sl.err, DEV_OK, code);
}

__device__ __forceinline__ int team() { return threadIdx.x / TM; }
__device__ __forceinline__ int team_thread() { return threadIdx.x % TM; }
__device__ __forceinline__ void team_sync() { asm volatile("bar.sync %0, %1;" ::"r"(2 + team()), "n"(TM) : "memory"); }
__device__ __forceinline__ void tree_sync() { asm volatile("bar.sync 1, %0;" ::"n"(TT) : "memory"); }
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// rows x cols block (ld rows) into shared memory (ld rows | 1), by one team.
__device__ __forceinline__ void stage(double* s, const double* g, int rows, int cols) {
  const int ld = rows | 1;
  for (int c = team_thread() >> 5; c < cols; c += TM / 32)
    for (int l = threadIdx.x & 31; l < rows; l += 32)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(s + l + c * ld)),
                   "l"(g + l + (int64_t)c * rows)
                   : "memory");
}

// Lines of a generator block into L2, a thread a line.
__device__ __forceinline__ void prefetch(const double* p, int64_t elems) {
  for (int64_t e = (int64_t)threadIdx.x * 16; e < elems; e += TT * 16)
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p + e));
}

// Sum over the L lanes of an output.  NC = 4: halves of the columns change hands (2 +
// 1 additions, then one a step, instead of 4 a step), and acc[0] is column own<4>(s);
// otherwise every lane has every column's.
template <int NC, int L>
__device__ __forceinline__ void sum_lanes(double (&acc)[NC], int s) {
  if constexpr (NC == 4) {
    const bool up = s & (L / 2), up2 = s & (L / 4);
    double a = up ? acc[2] : acc[0], b = up ? acc[3] : acc[1];
    const double oa = up ? acc[0] : acc[2], ob = up ? acc[1] : acc[3];
    a += __shfl_xor_sync(0xffffffffu, oa, L / 2);
    b += __shfl_xor_sync(0xffffffffu, ob, L / 2);
    double c = up2 ? b : a;
    const double oc = up2 ? a : b;
    c += __shfl_xor_sync(0xffffffffu, oc, L / 4);
    if (L == 8) c += __shfl_xor_sync(0xffffffffu, c, 1);
    acc[0] = c;   // column (s & L / 2 ? 2 : 0) + (s & L / 4 ? 1 : 0)
  } else {
#pragma unroll
    for (int q = 0; q < NC; ++q)
#pragma unroll
      for (int o = L / 2; o > 0; o >>= 1) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o);
  }
}

// One term of a small product: y(o, q) += sum_k m(o, k) x(k, q), m(o, k) at
// M + o * so + k * sk, x(k, q) at x + k + q * ldx in shared memory.
struct Term {
  const double* M;
  int so, sk, K;
  const double* x;
};

// Small product over a team, NS terms added up: lane s of an output's L takes
// k = s, s + L, ..., with NS * U loads of m in flight.  epi(o, q, sum) runs once
// per output and column.  L = 8 spreads the loads of long sums; four lanes are
// enough for the chains' steps (at most 64 terms from shared memory), and save a
// round of additions.
template <int NC, int NS, int U, int L, class Epi>
__device__ __forceinline__ void dotl(int no, const Term (&t)[NS], int ldx, Epi epi) {
  const int s = threadIdx.x % L, oo = team_thread() / L;
  int K = t[0].K;
  if (NS > 1) K = max(K, t[NS - 1].K);
  for (int o0 = 0; o0 < no; o0 += TM / L) {
    if (o0 + oo / (32 / L) * (32 / L) >= no) continue;   // the whole warp
    const int o = o0 + oo, oc = min(o, no - 1);
    double acc[NC];
#pragma unroll
    for (int q = 0; q < NC; ++q) acc[q] = 0.0;
    const double *p[NS], *x[NS];
#pragma unroll
    for (int j = 0; j < NS; ++j) {
      p[j] = t[j].M + (int64_t)oc * t[j].so + s * t[j].sk;
      x[j] = t[j].x + s;
    }
    for (int kb = 0; kb < K; kb += L * U) {
      double v[NS][U];
      bool full = true;
#pragma unroll
      for (int j = 0; j < NS; ++j) full = full && kb + L * U <= t[j].K;
      if (full) {
#pragma unroll
        for (int j = 0; j < NS; ++j)
#pragma unroll
          for (int u = 0; u < U; ++u) v[j][u] = p[j][L * u * t[j].sk];
#pragma unroll
        for (int j = 0; j < NS; ++j)
#pragma unroll
          for (int u = 0; u < U; ++u)
#pragma unroll
            for (int q = 0; q < NC; ++q) acc[q] = fma(v[j][u], x[j][L * u + q * ldx], acc[q]);
      } else {
#pragma unroll
        for (int j = 0; j < NS; ++j)
#pragma unroll
          for (int u = 0; u < U; ++u) v[j][u] = kb + L * u + s < t[j].K ? p[j][L * u * t[j].sk] : 0.0;
#pragma unroll
        for (int j = 0; j < NS; ++j)
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (kb + L * u < t[j].K) {
#pragma unroll
              for (int q = 0; q < NC; ++q)
                acc[q] = fma(v[j][u], kb + L * u + s < t[j].K ? x[j][L * u + q * ldx] : 0.0, acc[q]);
            }
      }
#pragma unroll
      for (int j = 0; j < NS; ++j) {
        p[j] += L * U * t[j].sk;
        x[j] += L * U;
      }
    }
    sum_lanes<NC, L>(acc, s);
    if (o < no) {
      if constexpr (NC == 4) {
        if (L == 4 || !(s & 1)) epi(o, (s & (L / 2) ? 2 : 0) + (s & (L / 4) ? 1 : 0), acc[0]);
      } else {
#pragma unroll
        for (int q = 0; q < NC; ++q)
          if (s == q) epi(o, q, acc[q]);
      }
    }
  }
}

// One row of A x (a lane a row, A at the lane's row: any valid one where the row
// does not count) for NC columns; lane k of the warp loads x(k, q) and passes it round.
// The terms are added up in runs of U, and the runs' sums one after the other.  One
// chain has more rounding error (n = 8192, rms in units of roundoff: leaves of 128 rows
// 3.4 against 1.6, of 40 rows 1.83 against 1.25; the kernel before this one, with
// several threads a row, 1.6 to 1.9 and 1.23), and saves 2.7 of 66 us at n = 65536, r = 1.
template <int NC, int U = 16, class X>
__device__ __forceinline__ void rows32(double (&acc)[NC], const double* A, int64_t lda, int K, X x) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int q = 0; q < NC; ++q) acc[q] = 0.0;
  for (int k0 = 0; k0 < K; k0 += 32) {
    const int kn = min(32, K - k0);
    double w[NC];
#pragma unroll
    for (int q = 0; q < NC; ++q) w[q] = lane < kn ? x(k0 + lane, q) : 0.0;
#pragma unroll
    for (int u0 = 0; u0 < 32; u0 += U) {
      if (u0 >= kn) break;
      double v[U], run[NC];
#pragma unroll
      for (int q = 0; q < NC; ++q) run[q] = 0.0;
      if (u0 + U <= kn) {
#pragma unroll
        for (int u = 0; u < U; ++u, A += lda) v[u] = __ldg(A);
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int q = 0; q < NC; ++q) run[q] = fma(v[u], __shfl_sync(0xffffffffu, w[q], u0 + u), run[q]);
      } else {
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = u0 + u < kn ? __ldg(A + u * lda) : 0.0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (u0 + u >= kn) break;
#pragma unroll
          for (int q = 0; q < NC; ++q) run[q] = fma(v[u], __shfl_sync(0xffffffffu, w[q], u0 + u), run[q]);
        }
      }
#pragma unroll
      for (int q = 0; q < NC; ++q) acc[q] += run[q];
    }
  }
}

__device__ __forceinline__ void col_norm(double* cn, double v) {
  v *= v;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0 && v != 0.0) atomicAdd(cn, v);
}

// Leaf-product unit u (leaf, piece, chunk) by one warp: 32 rows of
// C = alpha D B + beta Y (a single-leaf tree: the whole product, column norms
// included), then the (leaf, chunk) counter.
template <int NC>
__device__ void leaf_unit(const FlatArgs& a, int u) {
  const int per = a.npiece * a.nchunk, t = u / per, ch = u % a.nchunk, lane = threadIdx.x & 31;
  const Task tk = a.leaves[t];
  const Slot& sl = a.slots[tk.slot];
  const Node& nd = a.nodes[tk.node];
  const int j0 = ch * NC, m = nd.gm, n = nd.gn, r0 = (u % per) / a.nchunk * PR, nc = min(NC, sl.r - j0);
  if (nc > 0 && r0 < m) {
    const bool on = r0 + lane < m;
    const double* X = sl.B + nd.col0 + (int64_t)j0 * sl.ldb;
    const int64_t ldb = sl.ldb;
    double acc[NC];
    auto x = [&](int k, int q) { return q < nc ? __ldg(X + k + q * ldb) : 0.0; };
    const double* D = nd.D + min(r0 + lane, m - 1);
    if (n > 64) rows32<NC>(acc, D, m, n, x);
    else rows32<NC, 8>(acc, D, m, n, x);   // short rows have runs enough only of eight
    const double* Y = sl.Y ? sl.Y + nd.row0 + r0 + lane + (int64_t)j0 * sl.ldy : nullptr;
    const bool yterm = sl.beta != 0.0 && Y != nullptr;
    double* C = sl.C + nd.row0 + r0 + lane + (int64_t)j0 * sl.ldc;
#pragma unroll
    for (int q = 0; q < NC; ++q) {
      if (q >= nc) break;
      double v = 0.0;
      if (on) {
        v = sl.alpha * acc[q];
        if (yterm) v += sl.beta * __ldcg(Y + (int64_t)q * sl.ldy);
        C[(int64_t)q * sl.ldc] = v;
      }
      if (nd.root && sl.colnorm2) col_norm(sl.colnorm2 + j0 + q, v);
    }
  }
  __syncwarp();
  if (lane == 0) {
    __threadfence();
    atomicAdd(&a.dcnt[t * a.nchunk + ch], 1u);
  }
}

// A warp's next leaf-product unit, or -1.
__device__ __forceinline__ int claim_leaf(const FlatArgs& a) {
  const uint32_t nd = (uint32_t)(a.nleaves * a.npiece * a.nchunk);
  uint32_t u = nd;
  if ((threadIdx.x & 31) == 0 && ld_vol(&a.state[FL_D]) < nd) u = atomicAdd(&a.state[FL_D], 1u);
  u = __shfl_sync(0xffffffffu, u, 0);
  return u < nd ? (int)u : -1;
}

// Waits until n units are counted (tree warps; bounded: DEV_TIMEOUT, then on).
__device__ void wait_count(const FlatArgs& a, const uint32_t* ctr, uint32_t n) {
  if (threadIdx.x == 0) {
    uint32_t polls = 0;
    while (ld_acq(ctr) < n) {
      if (++polls > a.idle_limit) {
        set_err(a.slots[0], DEV_TIMEOUT);
        break;
      }
      __nanosleep(32);
    }
  }
  tree_sync();
}

// A finished unit of phase A or B: its writes published, then counted.
__device__ __forceinline__ void count_unit(uint32_t* ctr) {
  tree_sync();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(ctr, 1u);
  }
}

// Shared memory of the tree warps: a group, its nodes and the links of its path
// (depths 1 .. depth of its root).
struct FlatSmem {
  int64_t cur;   // the group held, -1: none
  FlatGroup g;
  Node nd[GN];
  FlatLink lk[kFlatDep];
};

__device__ void load_group(const FlatArgs& a, int gi, FlatSmem& S) {
  constexpr int GW = sizeof(FlatGroup) / 8, NW = sizeof(Node) / 8, LW = sizeof(FlatLink) / 8;
  if (S.cur == gi) return;   // (a block with one group loads it once)
  tree_sync();   // the unit before
  for (int e = threadIdx.x; e < GW; e += TT) ((uint64_t*)&S.g)[e] = __ldg((const unsigned long long*)&a.groups[gi] + e);
  tree_sync();
  if (threadIdx.x == 0) S.cur = gi;
  const int nw = S.g.nn * NW;
  for (int e = threadIdx.x; e < nw + S.g.depth * LW; e += TT) {
    const int l = e - nw;
    if (l < 0)
      ((uint64_t*)S.nd)[e] = __ldg((const unsigned long long*)&a.nodes[S.g.node[e / NW]] + e % NW);
    else
      ((uint64_t*)&S.lk[1])[l] = __ldg((const unsigned long long*)&a.links[S.g.path[l / LW]] + l % LW);
  }
  tree_sync();
}

// The B-terms of a group's nodes by warps of a team, 32 rows a job: G of the sibling
// = B Z, its rows of the workspace.  The group's root first.
template <int NC>
__device__ __forceinline__ void bterms(const Slot& sl, const FlatSmem& S, const double* Z, int km, int j0, int nc) {
  const FlatGroup& g = S.g;
  const int lane = threadIdx.x & 31, kk = km * NC;
  int job = team_thread() >> 5;
  for (int e = 0; e <= 2 * (g.nn - g.nl); ++e) {
    const int b = (e - 1) >> 1, c = (e - 1) & 1;   // child c of branch b
    const FlatLink& L = S.lk[g.depth];
    const Node& p = S.nd[g.nl + max(b, 0)];
    const int i = e == 0 ? g.nn - 1 : c ? g.right[b] : g.left[b];
    const double* B = e == 0 ? L.B : c ? p.B12 : p.B21;
    const int ks = e == 0 ? L.sku : p.cku[c ^ 1], kv = e == 0 ? L.kv : p.ckv[c];
    const int nrb = (ks + 31) / 32;
    if (job < nrb) {
      double* G = (double*)sl.ws + (e == 0 ? L.swf : p.cwf[c ^ 1]) + (int64_t)j0 * sl.ldws;
      for (; job < nrb; job += TM / 32) {
        const int r = job * 32 + lane;
        double acc[NC];
        rows32<NC>(acc, B + min(r, ks - 1), ks, kv, [&](int k, int q) { return Z[i * kk + k + q * km]; });
#pragma unroll
        for (int q = 0; q < NC; ++q)
          if (r < ks && q < nc) G[r + (int64_t)q * sl.ldws] = acc[q];
      }
    }
    job -= nrb;
  }
}

// Phase A unit: see the head of the file.
template <int NC>
__device__ void group_up(const FlatArgs& a, int gi, int ch, FlatSmem& S, double* sm) {
  load_group(a, gi, S);
  const FlatGroup& g = S.g;
  const Slot& sl = a.slots[g.slot];
  const int j0 = ch * NC, nc = min(NC, sl.r - j0), km = a.km, kk = km * NC, D = g.depth;
  if (nc <= 0) return;
  double* Z = sm;                        // the nodes' Z
  double* cur = Z + (g.nn - 1) * kk;     // the group root's, then the chain's
  double* const ring = sm + (GN + 2 + a.dep) * kk;
  const int rsz = (km | 1) * km, nb = a.nbuf;
  for (int i = 0; i < g.nl; ++i) prefetch(S.nd[i].V, (int64_t)S.nd[i].gn * S.nd[i].kv);
  auto stage_w = [&](int d) {
    if (d >= 2) stage(ring + d % nb * rsz, S.lk[d].W, S.lk[d].kv, S.lk[d].kpv);
    cp_commit();
  };
  const int tm = team();
  if (tm == 0) {
    stage_w(D);
    if (nb == 3) stage_w(D - 1);
  }
  for (int i = g.nl; i < g.nn; ++i) {
    const Node& x = S.nd[i];
    prefetch(x.W1, (int64_t)x.ckv[0] * x.kv);
    prefetch(x.W2, (int64_t)x.ckv[1] * x.kv);
    prefetch(x.B12, (int64_t)x.cku[0] * x.ckv[1]);
    prefetch(x.B21, (int64_t)x.cku[1] * x.ckv[0]);
  }
  double* const xs = sm + (GN + 2 + a.dep) * kk + nb * rsz + tm * a.nleaf * NC;
  for (int i = tm; i < g.nl; i += 2) {
    const Node& x = S.nd[i];
    const double* X = sl.B + x.col0 + (int64_t)j0 * sl.ldb;
    const int n = x.gn;
    team_sync();
    for (int l = team_thread(); l < n; l += TM)
#pragma unroll
      for (int q = 0; q < NC; ++q) xs[l + q * n] = q < nc ? __ldg(X + l + (int64_t)q * sl.ldb) : 0.0;
    team_sync();
    double* z = Z + i * kk;
    const Term t[1] = {{x.V, n, 1, n, xs}};
    dotl<NC, 1, 8, 8>(x.kv, t, n, [&](int o, int q, double v) { z[o + q * km] = v; });
  }
  for (int i = g.nl; i < g.nn; ++i) {
    const int b = i - g.nl;
    if (g.level[b]) tree_sync();   // children of the level below
    if ((b & 1) != tm) continue;
    const Node& x = S.nd[i];
    double* z = Z + i * kk;
    const Term t[2] = {{x.W1, x.ckv[0], 1, x.ckv[0], Z + g.left[b] * kk},
                       {x.W2, x.ckv[1], 1, x.ckv[1], Z + g.right[b] * kk}};
    dotl<NC, 2, 4, 8>(x.kv, t, km, [&](int o, int q, double v) { z[o + q * km] = v; });
  }
  tree_sync();
  if (tm == 0) {   // the chain to the branches above
    for (int d = D; d >= 2; --d) {
      if (nb == 3) cp_wait<1>();
      else cp_wait<0>();
      team_sync();
      stage_w(d - (nb - 1));
      const FlatLink& L = S.lk[d];
      const double* Ws = ring + d % nb * rsz;
      const int ldw = L.kv | 1;
      double* nxt = sm + (GN + (d & 1)) * kk;
      double* dst = a.ctb + ((int64_t)((d - 1) * a.ngroup + gi) * a.nchunk + ch) * kk;
      const Term t[1] = {{Ws, ldw, 1, L.kv, cur}};
      dotl<NC, 1, 8, 4>(L.kpv, t, km, [&](int o, int q, double v) {
        nxt[o + q * km] = v;
        dst[o + q * km] = v;
      });
      cur = nxt;
    }
    cp_wait<0>();
  } else {         // the B-terms of the group's nodes
    bterms<NC>(sl, S, Z, km, j0, nc);
  }
  // what phase C reads first
  for (int i = 0; i < g.nl; ++i) prefetch(S.nd[i].U, (int64_t)S.nd[i].gm * S.nd[i].ku);
  for (int i = g.nl; i < g.nn; ++i) {
    const Node& x = S.nd[i];
    prefetch(x.R1, (int64_t)x.cku[0] * x.ku);
    prefetch(x.R2, (int64_t)x.cku[1] * x.ku);
  }
}

// Phase B unit: Z of a branch from its groups' contributions, then its B-term.  The
// first part, before the contributions are there: B into the ring's slot 1.
__device__ void branch_pre(const FlatArgs& a, int bi, double* ring, FlatBranch& br, FlatLink& lk) {
  br = a.branches[bi];
  lk = a.links[br.node];
  tree_sync();   // the unit before
  if (team() == 0) stage(ring + (a.km | 1) * a.km, lk.B, lk.sku, lk.kv);
  cp_commit();
}
template <int NC>
__device__ void branch_z(const FlatArgs& a, const FlatBranch& br, const FlatLink& lk, int ch, double* sm,
                         const double* ring) {
  const Slot& sl = a.slots[br.slot];
  const int j0 = ch * NC, nc = min(NC, sl.r - j0), km = a.km, kk = km * NC;
  const int kv = lk.kv, sku = lk.sku;
  cp_wait<0>();
  if (nc <= 0) return;
  const double* src = a.ctb + ((int64_t)(lk.depth * a.ngroup + br.g0) * a.nchunk + ch) * kk;
  const int64_t gstride = (int64_t)a.nchunk * kk;
  // a warp takes four outputs, eight lanes the groups of each
  const int s = threadIdx.x & 7;
  for (int e = threadIdx.x >> 3; e < (kv * NC + 3) / 4 * 4; e += TT / 8) {
    const int c = e % kv, q = e / kv;
    const bool on = e < kv * NC;
    double acc[1] = {0.0};
    for (int g0 = s; on && g0 < br.gn; g0 += 64) {
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = g0 + 8 * u < br.gn ? __ldcg(src + (g0 + 8 * u) * gstride + c + q * km) : 0.0;
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (g0 - s + 8 * u < br.gn) acc[0] += v[u];
    }
    __syncwarp();
    sum_lanes<1, 8>(acc, s);
    if (on && s == 0) sm[c + q * km] = acc[0];
  }
  tree_sync();
  if (team() == 0) {
    const double* Bs = ring + (km | 1) * km;
    const int ldb = sku | 1;
    double* G = (double*)sl.ws + lk.swf + (int64_t)j0 * sl.ldws;
    const int64_t ld = sl.ldws;
    const Term t[1] = {{Bs, 1, ldb, kv, sm}};
    dotl<NC, 1, 8, 4>(sku, t, km, [&](int o, int q, double v) {
      if (q < nc) G[o + q * ld] = v;
    });
  }
}

// The translators R of depths 2 (and 3) of the path into the ring, by team 0.
__device__ __forceinline__ void stage_r(const FlatSmem& S, int d, double* ring, int km, int nb) {
  if (team() != 0) return;
  if (d <= S.g.depth) stage(ring + d % nb * ((km | 1) * km), S.lk[d].R, S.lk[d].ku, S.lk[d].kpu);
  cp_commit();
}

// Phase C unit.  staged: the first translators are on their way.
template <int NC>
__device__ void group_down(const FlatArgs& a, int gi, int ch, FlatSmem& S, double* sm, bool staged) {
  load_group(a, gi, S);
  const FlatGroup& g = S.g;
  const Slot& sl = a.slots[g.slot];
  const int j0 = ch * NC, nc = min(NC, sl.r - j0), km = a.km, kk = km * NC, D = g.depth;
  if (nc <= 0) return;
  tree_sync();   // the unit before
  double* F = sm;                               // the nodes' G, then F
  double* const Gs = sm + (GN + 2) * kk;        // G of the path: depth d at Gs + d kk (1 <= d < D)
  double* const ring = sm + (GN + 2 + a.dep) * kk;
  const int rsz = (km | 1) * km, nb = a.nbuf;
  if (!staged) {
    stage_r(S, 2, ring, km, nb);
    if (nb == 3) stage_r(S, 3, ring, km, nb);
  }
  const double* ws = (const double*)sl.ws + (int64_t)j0 * sl.ldws;
  const int64_t ld = sl.ldws;
  for (int e0 = threadIdx.x; e0 < (D - 1 + g.nn) * kk; e0 += 4 * TT) {
    double v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = e0 + u * TT, b = e / kk, i = (e % kk) % km, q = (e % kk) / km;
      v[u] = 0.0;
      if (b < D - 1 + g.nn) {
        const int64_t wf = b < g.nn ? S.nd[b].wf : S.lk[1 + b - g.nn].wf;
        const int ku = b < g.nn ? S.nd[b].ku : S.lk[1 + b - g.nn].ku;
        if (i < ku && q < nc) v[u] = __ldcg(ws + wf + i + q * ld);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = e0 + u * TT, b = e / kk;
      if (b < D - 1 + g.nn) (b < g.nn ? F + b * kk : Gs + (1 + b - g.nn) * kk)[e % kk] = v[u];
    }
  }
  tree_sync();
  // down the path: F at depth 1 is G
  if (team() == 0) {
    const double* f = D == 1 ? F + (g.nn - 1) * kk : Gs + kk;
    for (int d = 2; d <= D; ++d) {
      if (nb == 3) cp_wait<1>();
      else cp_wait<0>();
      team_sync();
      stage_r(S, d + nb - 1, ring, km, nb);
      const FlatLink& L = S.lk[d];
      const double* Rs = ring + d % nb * rsz;
      const int ldr = L.ku | 1;
      const double* G = d < D ? Gs + d * kk : F + (g.nn - 1) * kk;
      double* out = d < D ? sm + (GN + (d & 1)) * kk : F + (g.nn - 1) * kk;
      const Term t[1] = {{Rs, 1, ldr, L.kpu, f}};
      dotl<NC, 1, 8, 4>(L.ku, t, km, [&](int o, int q, double v) { out[o + q * km] = v + G[o + q * km]; });
      f = out;
    }
    cp_wait<0>();
  }
  // inside the group, a warp 32 rows of a child
  const int lane = threadIdx.x & 31;
  for (int i = g.nn - 1, job = 0; i >= g.nl; --i) {
    const int b = i - g.nl;
    if (i == g.nn - 1 || g.level[b + 1]) {
      tree_sync();
      job = threadIdx.x >> 5;
    }
    const Node& x = S.nd[i];
    const double* fp = F + i * kk;
    for (int c = 0; c < 2; ++c) {
      const int kc = x.cku[c], nrb = (kc + 31) / 32;
      double* fc = F + (c ? g.right[b] : g.left[b]) * kk;
      for (; job < nrb; job += TT / 32) {
        const int r = job * 32 + lane;
        double acc[NC];
        rows32<NC>(acc, (c ? x.R2 : x.R1) + min(r, kc - 1), kc, x.ku, [&](int k, int q) { return fp[k + q * km]; });
#pragma unroll
        for (int q = 0; q < NC; ++q)
          if (r < kc) fc[r + q * km] += acc[q];
      }
      job -= nrb;
    }
  }
  tree_sync();
  // C += alpha U F, a warp 32 rows of a leaf, once the leaf's pieces are done
  int job = threadIdx.x >> 5;
  for (int i = 0; i < g.nl; ++i) {
    const Node& x = S.nd[i];
    const int nrb = (x.gm + PR - 1) / PR;
    for (; job < nrb; job += TT / 32) {
      const int r = job * PR + lane;
      const bool on = r < x.gm;
      const double* fl = F + i * kk;
      const uint32_t* cnt = a.dcnt + (g.t0 + i) * a.nchunk + ch;
      uint32_t polls = 0;
      for (;;) {
        uint32_t done = 0;
        if (lane == 0) done = ld_acq(cnt) >= (uint32_t)a.npiece;
        if (__shfl_sync(0xffffffffu, done, 0)) break;
        const int u = claim_leaf(a);
        if (u >= 0) {
          leaf_unit<NC>(a, u);
        } else if (++polls > a.idle_limit) {
          if (lane == 0) set_err(a.slots[0], DEV_TIMEOUT);
          break;
        } else {
          __nanosleep(32);
        }
      }
      double* C = sl.C + x.row0 + r + (int64_t)j0 * sl.ldc;
      double cv[NC], acc[NC];
#pragma unroll
      for (int q = 0; q < NC; ++q) cv[q] = on && q < nc ? __ldcg(C + (int64_t)q * sl.ldc) : 0.0;
      rows32<NC>(acc, x.U + min(r, x.gm - 1), x.gm, x.ku, [&](int k, int q) { return fl[k + q * km]; });
#pragma unroll
      for (int q = 0; q < NC; ++q) {
        if (q >= nc) break;
        const double v = cv[q] + sl.alpha * acc[q];
        if (on) C[(int64_t)q * sl.ldc] = v;
        if (sl.colnorm2) col_norm(sl.colnorm2 + j0 + q, on ? v : 0.0);
      }
    }
    job -= nrb;
  }
}

template <int NC>
__global__ void __launch_bounds__(FT, 1) pmv_flat_kernel(FlatArgs a) {
  extern __shared__ __align__(16) unsigned char flat_smem[];
  FlatSmem& S = *(FlatSmem*)flat_smem;
  double* sm = (double*)(flat_smem + sizeof(FlatSmem));
  const int na = a.ngroup * a.nchunk, nb = a.nbranch * a.nchunk, blk = blockIdx.x, grid = gridDim.x;
  if (threadIdx.x < TT && blk < na) {
    double* const ring = sm + (GN + 2 + a.dep) * a.km * NC;
    if (threadIdx.x == 0) S.cur = -1;
    tree_sync();
    for (int u = blk; u < na; u += grid) {
      group_up<NC>(a, u / a.nchunk, u % a.nchunk, S, sm);
      count_unit(&a.state[FL_AFIN]);
    }
    // one group a block: what the next phases read is staged before the waits
    const bool one = na <= grid;
    if (one) {
      stage_r(S, 2, ring, a.km, a.nbuf);
      if (a.nbuf == 3) stage_r(S, 3, ring, a.km, a.nbuf);
    }
    FlatBranch br{};
    FlatLink lk{};
    if (blk < nb) branch_pre(a, blk / a.nchunk, ring, br, lk);
    wait_count(a, &a.state[FL_AFIN], (uint32_t)na);
    if (nb > 0) {
      for (int u = blk; u < nb; u += grid) {
        if (u != blk) branch_pre(a, u / a.nchunk, ring, br, lk);
        branch_z<NC>(a, br, lk, u % a.nchunk, sm, ring);
        count_unit(&a.state[FL_BFIN]);
      }
      wait_count(a, &a.state[FL_BFIN], (uint32_t)nb);
    }
    for (int u = blk; u < na; u += grid) group_down<NC>(a, u / a.nchunk, u % a.nchunk, S, sm, one);
  }
  for (int u; (u = claim_leaf(a)) >= 0;) leaf_unit<NC>(a, u);
  __shared__ int s_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(&a.state[FL_DONE], 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (s_last) {   // the last block out resets the counters
    for (int i = threadIdx.x; i < a.nleaves * a.nchunk; i += FT) a.dcnt[i] = 0;
    if (threadIdx.x == 0) {
      a.state[FL_AFIN] = 0;
      a.state[FL_BFIN] = 0;
      a.state[FL_D] = 0;
      __threadfence();
      a.state[FL_DONE] = 0;
    }
  }
}

size_t flat_bytes(int nleaf, int km, int dep, int nc, int nbuf) {
  return sizeof(FlatSmem) +
         sizeof(double) * ((size_t)(GN + 2 + dep) * km * nc + (size_t)nbuf * (km | 1) * km + 2 * (size_t)nleaf * nc);
}
constexpr size_t kFlatSmemCap = 220 * 1024;

// Groups and chunks of a product of r columns: the smallest groups that give no more
// units than SMs with chunks of four columns, then the narrowest chunks that do.  A
// unit's FP64 work has an SM to itself, so units beyond the SMs take a second pass
// over the tree's chain, and fewer leave SMs without a chain to carry.
struct FlatShape {
  int level, nc, nchunk;
};
FlatShape flat_shape(const FlatTables& f, int r, int sms) {
  FlatShape s;
  const int wide = (r + kFlatCw - 1) / kFlatCw;
  s.level = 0;
  while (s.level < kFlatLevels - 1 && (int64_t)f.lev[s.level].ngroup * wide > sms) ++s.level;
  s.nchunk = wide;
  while (s.nchunk < r && (int64_t)f.lev[s.level].ngroup * (s.nchunk + 1) <= sms) ++s.nchunk;
  s.nc = (r + s.nchunk - 1) / s.nchunk;
  s.nchunk = (r + s.nc - 1) / s.nc;
  return s;
}

}  // namespace

// Up to four columns in any case (n = 65536, k = 32: 68 / 115 / 160 / 210 us against
// the queued product's 156 / 187 / 215 / 235), more while the multiply-adds fit into
// the time that the chain leaves (n = 16384, 47 M: 155 against 194 us; n = 65536, 79 M:
// 245 against 265, but 455 against 362 at twice that; n = 20011, leaves of 156, 85 M:
// 255 against 203).  A second pass over the groups pays where the ranks are not small
// (n = 60000, k = 16, five columns: 197 against 226; n = 18944, k = 8, 20: 160 against 152).
bool pmv_flat_fits(const FlatTables& f, int64_t gen, int nleaf, int kmax, int rmax, int sms) {
  if (f.dep < 2 || f.dep > kFlatDep || rmax < 1 || rmax > kFlatCols || nleaf > 512 || kmax > 64 ||
      flat_bytes(nleaf, std::max(kmax, 1), f.dep, std::min(rmax, kFlatCw), 2) > kFlatSmemCap)
    return false;
  if (rmax <= 4) return true;
  const FlatShape s = flat_shape(f, rmax, sms);
  return gen * rmax <= 45000000 && (kmax >= 16 || (int64_t)f.lev[s.level].ngroup * s.nchunk <= sms);
}

uint32_t pmv_flat_levels(const FlatTables& f, int64_t gen, int nleaf, int kmax, int sms) {
  uint32_t levels = 0;
  for (int r = 1; r <= kFlatCols; ++r)
    if (pmv_flat_fits(f, gen, nleaf, kmax, r, sms)) levels |= 1u << flat_shape(f, r, sms).level;
  return levels;
}

// Estimated time in us: the chain's latency per pass over the groups, and 0.34 ns per
// multiply-add of an SM, its groups' tree part and its share of the leaf products
// (fitted to trees of 8 to 1024 leaves of 15 to 250 rows at 1 to 32 columns, within
// 25 %).
double pmv_flat_estimate(const FlatTables& f, int64_t nleaves, int64_t gen, int rmax, int sms) {
  const FlatShape s = flat_shape(f, rmax, sms);
  const double passes = std::ceil((double)f.lev[s.level].ngroup * s.nchunk / sms);
  const double tree = passes * (1 << s.level) * s.nc * (double)(gen - f.leaf_elems) / (double)nleaves;
  return 50.0 * passes - 15.0 + 0.34e-3 * (tree + (double)f.leaf_elems * rmax / sms);
}

void pmv_flat_space(const FlatTables& f, int64_t nleaves, int kmax, int rmax, int sms, int64_t* ctb, int64_t* counters) {
  const FlatShape s = flat_shape(f, rmax, sms);
  *ctb = std::max<int64_t>(1, (int64_t)f.lev[s.level].ngroup * f.dep * s.nchunk * std::max(kmax, 1) * s.nc);
  *counters = nleaves * s.nchunk;
}

cudaError_t launch_pmv_flat(const FlatTables& f, const Task* leaves, int64_t nleaves, const Slot* slots, int rmax,
                            int nleaf, int mleaf, int kmax, uint32_t* state, double* ctb, uint32_t* dcnt, int sms,
                            uint32_t idle_limit, cudaStream_t st) {
  if (nleaves <= 0) return cudaSuccess;
  const FlatShape shape = flat_shape(f, rmax, sms);
  const FlatLevel& lv = f.lev[shape.level];
  if (lv.ngroup > 0 && lv.groups == nullptr) return cudaErrorInvalidValue;
  FlatArgs a;
  a.leaves = leaves;
  a.nodes = f.nodes;
  a.links = f.links;
  a.groups = lv.groups;
  a.branches = lv.branches;
  a.slots = slots;
  a.state = state;
  a.ctb = ctb;
  a.dcnt = dcnt;
  a.nleaves = (int32_t)nleaves;
  a.ngroup = lv.ngroup;
  a.nbranch = lv.nbranch;
  a.nchunk = shape.nchunk;
  a.npiece = (std::max(mleaf, 1) + PR - 1) / PR;
  a.dep = f.dep;
  a.km = std::max(kmax, 1);
  a.nleaf = nleaf;
  a.idle_limit = idle_limit;
  const int nc = shape.nc;
  a.nbuf = flat_bytes(nleaf, a.km, f.dep, nc, 3) <= kFlatSmemCap ? 3 : 2;
  const size_t smem = flat_bytes(nleaf, a.km, f.dep, nc, a.nbuf);
  auto kern = nc == 1 ? pmv_flat_kernel<1> : nc == 2 ? pmv_flat_kernel<2> : nc == 3 ? pmv_flat_kernel<3> : pmv_flat_kernel<4>;
  static SmemOptIn opt_in[kFlatCw + 1];
  const cudaError_t e = opt_in[nc]((const void*)kern, kFlatSmemCap);
  if (e != cudaSuccess) return e;
  // one block an SM; with little work as many as have a group or a leaf piece per warp
  const int64_t pieces = nleaves * a.nchunk * a.npiece;
  const unsigned grid = (unsigned)std::min<int64_t>(
      sms, std::max<int64_t>({1, (int64_t)a.ngroup * a.nchunk, (pieces + 3) / 4}));
  void* args[] = {&a};
  return cudaLaunchCooperativeKernel((void*)kern, grid, FT, args, smem, st);
}

}  // namespace hss
