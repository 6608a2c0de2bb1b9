// How kq_qgemm_exact.cu cuts a call into tiles and K slices: host arithmetic, a pure function of the shapes and of how many
// clusters the device holds, shared by the launcher and a host program of the test suite.
#pragma once

#include <algorithm>
#include <cstdint>

namespace kq {
namespace exact {

#ifdef __CUDACC__
#define KQ_EXACT_FN __host__ __device__ constexpr
#else
#define KQ_EXACT_FN constexpr
#endif

// one binary16 part or two, one bf16 part or three, or int8 x int8
enum MathKind : int { kHalf1, kHalf2, kBf1, kBf3, kInt8 };
KQ_EXACT_FN uint32_t parts_of(int math) { return math == kBf3 ? 3u : math == kHalf2 ? 2u : 1u; }

constexpr uint32_t kMaxNT = 256;           // activation rows per tile
constexpr uint32_t kMaxClusterSplits = 4;  // K slices that meet in a cluster: two or four (eight CTAs, the portable most)

// Clocks of one k-step.  The conversion of the weights does not grow with the tile, its copy and the MMAs do; a
// drain costs its 32 to 256 fmas, 330 clocks at least, and is hidden until it alone fills the step; the two or three
// parts of f32 rows cost what their tiles take to arrive, and above 192 rows the power cap, the more of it the more pairs
// are at work: int4 group 32 f32, between k = 1,536 and 14,336, at 160, 192, 224, 256 rows 1,650, 1,590, 1,820, 1,910 on
// 37 pairs, 1,780, 1,760, 2,230, 2,340 on 64, 1,970, 1,940, 2,410, 2,520 on 74.  The price above 192 rows is that of calls
// whose last wave is not full (at 10 clocks a row 2048 x 14336 -> 4096 went from two waves of 256 rows, 543 us, to three of
// 160, 591).  Measured with 74 pairs between k = 4,096 and 8,192, at 1.92 GHz, nt = 32, 64, 96, 128, 160, 192, 224, 256:
//   int4, group 32   binary16 683, 798, 905, 1,048, 1,275, 1,450, 1,660, 1,750; f32 900, 1,200, 1,320, 1,510, 1,810,
//                    1,960, 2,370, 2,940
//   int8, tiled      binary16 535, 632, 632, 711, 764, 836, 950, 1,020 to 1,190; f32 780, 870, 890, 1,110, 1,290, 1,450,
//                    1,600, 2,070
//   int8, rows       (k = 4,096 to 12,288, 6 pairs; 32, 64, 128, 192, 256) binary16 625, 700, 835, 890, 985; f32 1,110, 1,325,
//                    1,415, 1,580, 1,675 (bytes take 9 instructions for four bf16 integers, 4 for binary16)
inline uint32_t kstep_clocks(uint32_t nt, int math, uint32_t drains_x4, bool int8_weights) {
  const bool int8 = math == kInt8, bytes_to_bf = int8_weights && (math == kBf1 || math == kBf3);
  const uint32_t parts = parts_of(math);
  const uint32_t mma = 4 * parts * std::max(nt / 2, 48u);
  const uint32_t step = int8 ? 650 + nt : 450 + (bytes_to_bf ? 200 : 0) + 100 * parts + nt + drains_x4 * (nt * 8 / 5 + 20) / 4;
  const uint32_t fill = parts == 3 ? (nt > 192 ? nt * 35 / 4 : 740 + nt * 28 / 5) : parts == 2 ? 640 + nt * 21 / 5 : 0;
  const uint32_t drain = int8 ? 0u : drains_x4 * std::max(nt * 7 / 2 + 60, 330u) / 4;
  return std::max({mma, step, fill, drain});
}

// k-steps of a call (128 bytes of activations each), k16 slices of its accumulator chains, and the k-steps that a K slice
// is a multiple of: it is a whole number of int4 chains (an int8 chain may end anywhere).  group: 0 for int8 weights.
struct Steps { uint32_t ksteps, drain16, slice_unit; };
inline Steps steps_of(uint32_t k, int math, uint32_t group, uint32_t max_chain) {
  const uint32_t step_k = math == kInt8 ? 128 : 64, drain16 = (group != 0 ? std::min(group, max_chain) : max_chain) / 16;
  return Steps{(k + step_k - 1) / step_k, drain16, group != 0 && drain16 > 4 ? drain16 / 4 : 1};
}

struct Geometry { uint32_t nt, m_tiles, splits, cluster_splits; uint64_t clocks; };  // clocks: what it is expected to take
// Tile width and K slices by estimated time: whole waves of pairs, each a fixed cost (tile fill, first
// loads, epilogue) plus its k-steps.  Two or four slices may meet in a cluster: no second launch and no partial sums in
// memory, but 33 clusters of two pairs and 15 of four are all the device holds (74 pairs by themselves), and they start
// later and wait for one another (priced at 750 clocks a slice, 153 x 1152 -> 5280 int8 binary16 went from 63 tiles, 11.3 us,
// to 21 clusters, 14.1).  Other slices add the reduce launch and the partial sums, written and read at 2,200 bytes per clock.
// The prices are those that come closest over 242 shapes (17 to 2,048 rows, all storages and activations) of which up to
// eighteen cuts each were timed: 0.5 % behind the fastest in the mean, more than 5 % on eight of them.
//   (us, with its split launch; reduce launch | cluster)  65 x 1152 -> 3072 group 16, four slices 16.0 | 13.8;
//   300 x 4096 -> 4096 int8 binary16, two 29.0 | 22.8; 100 x 2048 -> 2048 group 128, four 18.2 | 15.4;
//   333 x 8960 -> 1536, four, 72 tiles of 128 rows 45.4, 48 of 192 rows 49.3 | 46.6
// Widths between the powers of two: 804 x 4096 -> 6144 f32 at 160 rows 117, 128 152, 192 123, 256 148.
inline Geometry choose_geometry(uint32_t m, uint32_t n_total, uint32_t pairs, const Steps& of, int math, bool int8_weights, bool may_split,
                                const uint32_t (&slots)[kMaxClusterSplits + 1], uint64_t partial_room) {
  const uint32_t ksteps = of.ksteps, drain16 = of.drain16, slice_unit = of.slice_unit;
  Geometry best = {kMaxNT, (m + kMaxNT - 1) / kMaxNT, 1, 1, 0};
  uint64_t best_cost = ~0ull;
  const uint32_t drains_x4 = std::max(1u, 16 / drain16);  // accumulator chains per k-step, times four
  const uint32_t most = (m + 31) / 32;
  for (uint32_t mt = (m + kMaxNT - 1) / kMaxNT; mt <= most; ++mt) {
    uint32_t nt = ((m + mt - 1) / mt + 31) / 32 * 32;
    if ((m + nt - 1) / nt != mt) continue;
    const uint32_t per = kstep_clocks(nt, math, drains_x4, int8_weights);
    for (uint32_t splits = 1; splits <= (may_split ? 16u : 1u); splits *= 2) {
      if (splits > 1 && ksteps / splits < 4) break;
      uint32_t each = (ksteps + splits - 1) / splits;
      each = (each + slice_unit - 1) / slice_unit * slice_unit;
      for (uint32_t in_cluster = 0; in_cluster < 2; ++in_cluster) {
        if (in_cluster != 0 ? splits == 1 || splits > kMaxClusterSplits || slots[splits] == 0 || (ksteps + each - 1) / each != splits
                            : splits > 1 && static_cast<uint64_t>(splits) * m * n_total * 4 > partial_room)
          continue;
        const uint32_t room = in_cluster != 0 ? slots[splits] * splits : slots[1];
        const uint64_t waves = (static_cast<uint64_t>(pairs) * mt * splits + room - 1) / room;
        uint64_t cost = waves * (6000 + nt * 30 + static_cast<uint64_t>(each) * per + (in_cluster != 0 ? 2500 : 0));
        if (splits > 1 && in_cluster == 0) cost += 4400 + 140 * splits + static_cast<uint64_t>(m) * n_total * (2 * splits + 1) * 4 / 2200;
        if (cost < best_cost) {
          best_cost = cost;
          best = {nt, mt, splits, in_cluster != 0 ? splits : 1u, cost};
        }
      }
    }
    if (mt >= 8 * slots[1]) break;
  }
  return best;
}

// Most k of an accumulator chain.  Each of a chain's accumulations truncates (half a unit of 2^-24 on average, all the
// same way), while the sums of the drain round to nearest.  Relative error against f64 (2-norm, k = 4,096), and us for
// 300 x 4096 -> 4090 int8, with chains of 64, 128, 256 and 1,024:
//   f32, three parts        1.3, 2.7, 6.0, 26e-7   50, 47, 46, 46
//   f32, two parts (tiled)  1.7, 2.5, 4.8, 21e-7   (1024 x 4096 -> 4096) 68, 63, 61.5, 60
//   binary16, int8 weights  1.6, 1.5, 2.3, 9.7e-7  32, 30, 29, 29
//   bf16, int8 weights      1.1, 1.0, 1.1, 3.3e-7  44, 42, 41, 40
//   binary16, int4 weights  1.5, 1.1, 0.9, 2.1e-7  (300 x 8192 -> 4000) 52, 47, 45, 43
// An f32 multiply-add per weight is 2.1e-7 from f64 there, the int8 GEMV 8 to 13e-7: each is kept below the path it
// stands in for.
inline uint32_t chain_of(int math, bool int8_weights) {
  if (math == kBf3) return 64;
  return math == kHalf1 && int8_weights ? 128 : 256;
}

}  // namespace exact
}  // namespace kq
