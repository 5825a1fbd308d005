// Splitting a merged level list by size class (seg_split, hss_levels.h): the list's
// tasks name their matrix by slot, and every part's sizes are those of the nodes its
// tasks name, in whatever order the matrices come.  Prints one line per failure.
#include <cstdio>
#include <cstring>

#include "hss_levels.h"

using namespace hss;

int main() {
  // matrix i: three leaves of size[i] rows
  const int perms[][4] = {{128, 60, 60, 30}, {60, 128, 30, 60}, {30, 60, 60, 128}, {60, 60, 128, 128}, {128, 128, 60, 60}};
  for (const auto& size : perms) {
    std::vector<std::vector<Node>> nodes(4, std::vector<Node>(3));
    std::vector<Task> tasks(2);   // the list starts behind another one
    std::memset(tasks.data(), 0, 2 * sizeof(Task));
    Seg g;
    g.off = 2;
    for (int i = 0; i < 4; ++i)
      for (int l = 0; l < 3; ++l) {
        Node& x = nodes[i][l];
        std::memset(&x, 0, sizeof(x));
        x.leaf = 1;
        x.m = x.n = x.gm = x.gn = size[i];
        x.ku = x.kv = x.k = x.mr = x.nr = 8;
        x.mk = x.nk = size[i] - 8;
        tasks.push_back(Task{nullptr, l, i});
        seg_add(g, x, nodes[i].data());
      }
    seg_split(g, tasks, [&](int64_t i) { return nodes[tasks[g.off + i].slot].data(); });
    int64_t seen = 0;
    std::vector<int> got(12, 0);
    for (const Seg& p : g.parts) {
      if (p.off != g.off + seen) std::printf("a part starts at %d\n", (int)p.off);
      int mmax = 0, smin = INT32_MAX;
      for (int64_t t = p.off; t < p.off + p.cnt; ++t) {
        ++got[tasks[t].slot * 3 + tasks[t].node];
        mmax = std::max(mmax, size[tasks[t].slot]);
        smin = std::min(smin, size[tasks[t].slot]);
      }
      if (size_class(nodes[tasks[p.off].slot][0]) != size_class(nodes[tasks[p.off + p.cnt - 1].slot][0]))
        std::printf("a part of several classes\n");
      if (p.mmax != mmax || p.smin != smin)
        std::printf("sizes %d %d %d %d: a part of nodes of %d to %d rows has the sizes %d to %d\n", size[0], size[1],
                    size[2], size[3], smin, mmax, p.smin, p.mmax);
      seen += p.cnt;
    }
    if (seen != 12) std::printf("parts of %d tasks\n", (int)seen);
    for (int c : got)
      if (c != 1) std::printf("a task appears %d times\n", c);
  }
  return 0;
}
