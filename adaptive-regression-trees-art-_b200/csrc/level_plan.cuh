// level_plan.cuh -- how a level's nodes are dealt to the CTAs of its two launches
// (tree.cu); host code, plain C++.
#pragma once
#include <algorithm>
#include <cstdint>

namespace art {

constexpr int kLevelThreads = 256;
constexpr int kLevelWarps = kLevelThreads / 32;
constexpr int kMaxRanks = 16;      // CTAs of a cluster, and partial sums of a node, at most
constexpr int kSingleRows = 1024;  // one warp's node at most: 32 mask words, one partial sum

struct LevelPlan {
  int64_t count;
  int64_t joint;  // rows above which a node is a cluster's (-1: every node)
  int nodes;      // nodes a CTA of the first launch, a cluster of the second
  int single;     // rows up to which a node is one warp's (-1: none)
};

// Up to kLevelFew nodes: the second launch alone takes them all (one launch less,
// 6 to 9 us in place of 9 to 11).  Beyond, `joint` grows with the number of
// nodes: 100 single CTAs leave a third of the device idle, 300 fill it, and then a
// cluster is worth its barriers only for a node that would outlast the others (300
// nodes of 5,000 rows, d = 2: 21 us by CTAs, 85 by clusters; 307 nodes of 450 to
// 400,000 rows, d = 2 to 32: 0.84 ms with joint at 6,144 rows, 0.92 at 12,288;
// 1,000 nodes of 450 to 20,000 rows: 0.30 ms at 8,192 to 10,240, 0.38 at 20,480).
// 444 CTAs for the first launch (three an SM, all resident) until that is eight
// nodes each, which their warps take side by side; 148 clusters for the second:
// 296 cost levels of small nodes 2 to 4 us more, 74 the large ones 3 %.  (`ctas`: the
// first launch's where another kernel makes it.)
constexpr int64_t kLevelFew = 32;
inline int64_t level_joint(int64_t count) { return 2048 * std::min<int64_t>(std::max<int64_t>(count / 100, 1), 4); }
inline LevelPlan level_small(int64_t count, int ctas = 444) {
  LevelPlan L{count, level_joint(count), (int)std::min<int64_t>((count + ctas - 1) / ctas, 8), -1};
  if (L.nodes > 1) L.single = std::min(kSingleRows, 128 * L.nodes);
  return L;
}
inline LevelPlan level_large(int64_t count) {
  if (count <= kLevelFew) return LevelPlan{count, -1, 1, -1};
  return LevelPlan{count, level_joint(count), (int)std::min<int64_t>((count + 147) / 148, kLevelThreads), -1};
}

// CTAs of a cluster: the most that the device has room for, by fits(size).
template <typename F>
int level_cluster(F fits) {
  int c = kMaxRanks;
  while (c > 1 && !fits(c)) c /= 2;
  return c;
}

}  // namespace art
