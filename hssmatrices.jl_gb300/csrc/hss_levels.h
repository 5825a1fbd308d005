// Task lists by tree level, as the host launches them, and the key that a recorded
// launch sequence is kept under (hss_capi.cpp).
#pragma once
#include <algorithm>
#include <climits>
#include <cstdint>
#include <utility>
#include <vector>

#include "hss_internal.h"
#include "hss_launch.h"

namespace hss {

// A list of tasks, with the largest sizes of its nodes.  Every field shapes launches:
// a new one also goes into seg_key.
struct Seg {
  int64_t off = 0, cnt = 0;
  int mmax = 0, nmax = 0, kumax = 0, kvmax = 0;   // largest node of the list
  int c1u = 0, c2u = 0, c1v = 0, c2v = 0;          // largest children's ranks (branches)
  int kmax = 0, mkmax = 0;                         // largest ULV k and m - k
  int c1mr = 0, c2mr = 0, c1nr = 0, c2nr = 0;      // largest children's reduced sizes
  int64_t sv_stage = 0;                            // largest upward-solve staging need
  int mk_in = 0, rootmax = 0;                      // largest m - k of the nodes that are not roots; largest root
  int smin = INT32_MAX;                            // smallest node: its larger side
  bool leaves = false, branches = false;           // kinds of node in the list
  std::vector<Seg> parts;                          // the list by size of node (empty: one size class)
};

// Size class of a node for the factor and solve kernels, whose registers and
// shared memory are laid out for the largest node of a launch.
inline int size_class(const Node& x) {
  const int s = std::max(x.m, x.n);
  return s <= 32 ? 0 : s <= 64 ? 1 : s <= 96 ? 2 : s <= 128 ? 3 : s <= 256 ? 4 : 5;
}

// Counts node x (children in `nodes`) into the largest sizes of a list.
inline void seg_add(Seg& v, const Node& x, const Node* nodes) {
  ++v.cnt;
  v.smin = std::min(v.smin, std::max(x.m, x.n));
  v.mmax = std::max(v.mmax, x.m);
  v.nmax = std::max(v.nmax, x.n);
  v.kumax = std::max(v.kumax, x.ku);
  v.kvmax = std::max(v.kvmax, x.kv);
  v.kmax = std::max(v.kmax, x.root ? 0 : x.k);
  v.mkmax = std::max(v.mkmax, x.mk);
  if (x.root) v.rootmax = std::max(v.rootmax, x.m);
  else v.mk_in = std::max(v.mk_in, x.mk);
  (x.leaf ? v.leaves : v.branches) = true;
  const Node* a = x.leaf ? nullptr : &nodes[x.left];
  const Node* b = x.leaf ? nullptr : &nodes[x.right];
  v.sv_stage = std::max(v.sv_stage, solve_up_stage_need(x.m, x.k, x.mk, x.nk, x.kv, x.leaf, x.root, a ? a->mr : 0,
                                                        b ? b->mr : 0, a ? a->kv : 0, b ? b->kv : 0));
  if (x.leaf) return;
  v.c1u = std::max(v.c1u, a->ku);
  v.c2u = std::max(v.c2u, b->ku);
  v.c1v = std::max(v.c1v, a->kv);
  v.c2v = std::max(v.c2v, b->kv);
  v.c1mr = std::max(v.c1mr, a->mr);
  v.c2mr = std::max(v.c2mr, b->mr);
  v.c1nr = std::max(v.c1nr, a->nr);
  v.c2nr = std::max(v.c2nr, b->nr);
}

// The list v (tasks off .. off + cnt of `tasks`) ordered by size class, with a part
// per class where there are several; nodes(i): the node array of its i-th task, asked
// for before the tasks move (it may look at them).
template <class F>
void seg_split(Seg& v, std::vector<Task>& tasks, F&& nodes) {
  struct Item {
    int cls;
    Task task;
    const Node* nodes;
  };
  v.parts.clear();
  auto cls = [&](int64_t i) { return size_class(nodes(i)[tasks[v.off + i].node]); };
  int64_t same = 1;
  while (same < v.cnt && cls(same) == cls(0)) ++same;
  if (same >= v.cnt) return;
  std::vector<Item> items((size_t)v.cnt);
  for (int64_t i = 0; i < v.cnt; ++i) {
    const Node* nd = nodes(i);
    const Task& t = tasks[v.off + i];
    items[i] = Item{size_class(nd[t.node]), t, nd};
  }
  std::stable_sort(items.begin(), items.end(), [](const Item& a, const Item& b) { return a.cls < b.cls; });
  for (int64_t i = 0; i < v.cnt; ++i) {
    if (i == 0 || items[i].cls != items[i - 1].cls) {
      v.parts.emplace_back();
      v.parts.back().off = v.off + i;
    }
    tasks[v.off + i] = items[i].task;
    seg_add(v.parts.back(), items[i].nodes[items[i].task.node], items[i].nodes);
  }
}

// The task lists one launch sequence walks: a plan's own (slot = tree of the
// forest) or lists merged over several single-tree plans (slot = item).
struct Levels {
  const Task* d_tasks = nullptr;
  const std::vector<Seg>* by_h = nullptr;
  const std::vector<Seg>* by_d = nullptr;
  const std::vector<Seg>* mv_up = nullptr;
  const std::vector<Seg>* mv_dn = nullptr;
  Seg leaves;
  // persistent product: largest leaf columns / rows, largest rank, non-root nodes
  int nleaf = 0, mleaf = 0, kmax = 0;
  int64_t ntasks = 0;
  int64_t nodes_max = 0, nslots = 0;   // largest node array of a slot's plan; slots
  int64_t ninner = 0;                  // non-root branches
  int device = 0;
  FlatTables flat;   // flat product tables (dep = 0: not available)
  int64_t gen_len = 0;
  // translators to prefetch into L2 (FP64 and pair copies; null: none)
  const double* pf64 = nullptr;
  const float2* pfdf = nullptr;
  int64_t pf_elems = 0;
};

// A word mixed into a key.
inline uint64_t mix(uint64_t h, uint64_t v) {
  h = (h ^ v) * 0x9E3779B97F4A7C15ull;
  return h ^ (h >> 29);
}

// A list's share of a key: the list, its sizes, and its parts.
inline uint64_t seg_key(uint64_t h, const Seg& g) {
  for (int64_t x : {g.off, g.cnt, g.sv_stage}) h = mix(h, (uint64_t)x);
  for (int x : {g.mmax, g.nmax, g.kumax, g.kvmax, g.c1u, g.c2u, g.c1v, g.c2v, g.kmax, g.mkmax, g.c1mr, g.c2mr, g.c1nr,
                g.c2nr, g.mk_in, g.rootmax, g.smin, (int)g.leaves, (int)g.branches})
    h = mix(h, (uint64_t)(int64_t)x);
  h = mix(h, g.parts.size());
  for (const Seg& p : g.parts) h = seg_key(h, p);
  return h;
}

// Key of a launch sequence over task lists L with the device slot table `slots`: all
// that the launches take from L.  (The task buffer's contents are read when a recorded
// sequence runs, its lists' offsets and sizes are part of the recording: a batcher
// keeps its buffers' addresses from one batch to the next.)
inline uint64_t levels_key(const Levels& L, const void* slots, int64_t extra) {
  uint64_t h = 1469598103934665603ull;
  for (const void* p : {(const void*)L.d_tasks, slots, (const void*)L.pf64, (const void*)L.pfdf,
                        (const void*)L.flat.links})
    h = mix(h, (uint64_t)(uintptr_t)p);
  for (int64_t x : {extra, (int64_t)L.nleaf, (int64_t)L.mleaf, (int64_t)L.kmax, L.ntasks, L.nodes_max, L.nslots,
                    L.ninner, (int64_t)L.device, L.gen_len, L.pf_elems, (int64_t)L.flat.dep, L.flat.leaf_elems})
    h = mix(h, (uint64_t)x);
  h = seg_key(h, L.leaves);
  for (const std::vector<Seg>* v : {L.by_h, L.by_d, L.mv_up, L.mv_dn}) {
    h = mix(h, v->size());
    for (const Seg& g : *v) h = seg_key(h, g);
  }
  return h;
}

}  // namespace hss
