// The key of a recorded launch sequence (hss_levels.h) on merged task lists: two
// batches whose lists have the same offsets, counts and largest sizes, but other size
// classes, launch other kernels over other parts and need other keys.  Prints one line
// per failure.
#include <cstdio>
#include <cstring>

#include "hss_levels.h"

using namespace hss;

namespace {

Node leaf(int size, int k) {
  Node x;
  std::memset(&x, 0, sizeof(x));
  x.leaf = 1;
  x.m = x.n = x.gm = x.gn = size;
  x.ku = x.kv = x.k = x.nk = k;
  x.mk = size - k;
  x.nk = size - k;
  x.mr = x.nr = k;
  return x;
}

// One level of leaves of the given sizes.
uint64_t key(const std::vector<int>& sizes, int parts, const std::vector<Seg>* mv = nullptr, int mleaf = 0) {
  std::vector<Node> nodes;
  std::vector<Task> tasks;
  for (size_t i = 0; i < sizes.size(); ++i) {
    nodes.push_back(leaf(sizes[i], 16));
    tasks.push_back(Task{nullptr, (int32_t)i, 0});
  }
  Seg g;
  for (const Node& x : nodes) seg_add(g, x, nodes.data());
  seg_split(g, tasks, [&](int64_t) { return nodes.data(); });
  if ((int)g.parts.size() != parts) std::printf("parts %d\n", (int)g.parts.size());
  const std::vector<Seg> lists{g}, none;
  Levels L;
  L.by_h = L.by_d = &lists;
  L.mv_up = L.mv_dn = mv ? mv : &none;
  L.mleaf = mleaf;
  return levels_key(L, nullptr, 1);
}

#define EXPECT(c) \
  if (!(c)) std::printf("failed: %s\n", #c)

}  // namespace

int main() {
  EXPECT(key({128, 60, 60}, 2) == key({128, 60, 60}, 2));
  EXPECT(key({128, 60, 60}, 2) != key({128, 128, 60}, 2));   // one and two of the large class
  EXPECT(key({128, 96, 60}, 3) != key({128, 60, 60}, 2));    // another class
  EXPECT(key({128, 128, 128}, 0) != key({128, 128, 100}, 0)); // the smallest size decides the solve's kernel
  // the product's lists and sizes shape the refinement's launches
  std::vector<Seg> mv(1);
  mv[0].cnt = 3;
  EXPECT(key({128, 60}, 2) != key({128, 60}, 2, &mv));
  const uint64_t k3 = key({128, 60}, 2, &mv);
  mv[0].c1u = 8;
  EXPECT(k3 != key({128, 60}, 2, &mv));
  EXPECT(key({128, 60}, 2) != key({128, 60}, 2, nullptr, 128));
  return 0;
}
