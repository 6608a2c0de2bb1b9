// Host-side check of how the many-row linears cut a call (karume_b200/csrc/kq_exact_geometry.h).  Without an argument: over
// a grid of shapes, tiles cover the rows, no K slice is empty, slices that meet in a cluster fit one, and partial sums in
// memory fit the scratch.  With one: lines "m n k math group" (group 0: int8 weights) on standard input, and "rows-per-tile
// tiles slices slices-in-a-cluster" of each printed, for a device that holds 74 pairs, 33 clusters of two and 15 of four.
#include <cstdio>
#include <initializer_list>

#include "kq_exact_geometry.h"

using namespace kq::exact;

static const uint32_t kSlots[kMaxClusterSplits + 1] = {0, 74, 33, 0, 15};

static Steps steps(uint32_t k, int math, uint32_t group) { return steps_of(k, math, group, math == kInt8 ? 1024 : chain_of(math, group == 0)); }

static int check(uint32_t m, uint32_t n, uint32_t k, int math, uint32_t group, uint64_t room) {
  const Steps s = steps(k, math, group);
  const Geometry g = choose_geometry(m, n, (n + 255) / 256, s, math, group == 0, true, kSlots, room);
  const uint32_t each = ((s.ksteps + g.splits - 1) / g.splits + s.slice_unit - 1) / s.slice_unit * s.slice_unit;
  const char* why = nullptr;
  if (g.nt == 0 || g.nt > kMaxNT || g.nt % 32 != 0 || (m + g.nt - 1) / g.nt != g.m_tiles) why = "tiles";
  else if (g.cluster_splits != 1 && (g.cluster_splits != g.splits || g.splits > kMaxClusterSplits || kSlots[g.splits] == 0)) why = "cluster";
  else if (g.cluster_splits != 1 && (s.ksteps + each - 1) / each != g.splits) why = "an empty slice";
  else if (g.splits > 1 && g.cluster_splits == 1 && static_cast<uint64_t>(g.splits) * m * n * 4 > room) why = "scratch";
  if (why != nullptr) std::printf("FAIL %s: m=%u n=%u k=%u math=%d group=%u: %u %u %u %u\n", why, m, n, k, math, group, g.nt, g.m_tiles, g.splits, g.cluster_splits);
  return why != nullptr;
}

int main(int argc, char**) {
  if (argc > 1) {
    unsigned m, n, k, math, group;
    while (std::scanf("%u %u %u %u %u", &m, &n, &k, &math, &group) == 5) {
      const Geometry g = choose_geometry(m, n, (n + 255) / 256, steps(k, static_cast<int>(math), group), static_cast<int>(math), group == 0, true, kSlots, 256u << 20);
      std::printf("%u %u %u %u\n", g.nt, g.m_tiles, g.splits, g.cluster_splits);
    }
    return 0;
  }
  unsigned cases = 0;
  for (uint32_t m : {1u, 17u, 31u, 33u, 64u, 97u, 160u, 161u, 225u, 256u, 257u, 333u, 449u, 700u, 1024u, 1905u, 4096u, 20000u})
    for (uint32_t n : {1u, 16u, 112u, 257u, 1536u, 4096u, 8961u, 18944u, 151936u})
      for (uint32_t k : {16u, 64u, 576u, 1152u, 4096u, 8960u, 14336u})
        for (int math : {kHalf1, kHalf2, kBf1, kBf3, kInt8})
          for (uint32_t group : {0u, 16u, 32u, 128u, 4096u}) {
            if ((group != 0 && (k % group != 0 || math == kHalf2 || math == kInt8))) continue;
            for (uint64_t room : {uint64_t(0), uint64_t(1) << 20, uint64_t(1) << 28}) {
              if (check(m, n, k, math, group, room)) return 1;
              ++cases;
            }
          }
  std::printf("ok %u\n", cases);
  return 0;
}
