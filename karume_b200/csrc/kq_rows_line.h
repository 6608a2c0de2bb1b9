// Which kernel runs up to sixteen rows over one row-major packed weight: host arithmetic, a pure function of the shape, shared
// by the launchers and a host program of the test suite.  Estimates in units of 0.01 us, fitted to 1,309 timed calls (1 to
// 16 rows, 16 to 36,699 channels, k 64 to 12,288, int4 groups of 16 and 128 and int8, f32, binary16 and bf16; each within
// 6 to 9 % in the mean, and 1 % behind the faster side in the mean).  us, others | kq_qgemv_rows.cu:
//   the generic kernel stays for small calls  int4 2 x 256 -> 64 2.1 | 3.6, 1 x 512 -> 600 2.6 | 3.1, 3 x 512 -> 600 3.6 | 4.6,
//                                             3 x 256 -> 1024 2.6 | 4.6, but 1 x 8064 -> 82 12.8 | 5.2, int8 15.6 | 4.2
//   the many-row kernel, f32                  int4 group 128 1 x 768 -> 36699 21.0 | 9.8, 4 x 768 -> 36699 20.5 | 16.3, 2 x 4096 -> 4090
//                                             15.4 | 12.0, but 4 x 4096 -> 4090 14.9 | 18.5; int8 1 x 4096 -> 4090 16.9 | 8.7,
//                                             but 8 x 768 -> 36699 24.6 | 29.5
//   ... binary16, one launch less             int4 group 128 1 x 4096 -> 4090 11.6 | 8.7; int8 1 x 4096 -> 4090 10.8 | 7.7, but
//                                             2 x 4096 -> 2841 10.8 | 12.3, 4 x 2048 -> 3571 8.7 | 13.3, 16 x 8064 -> 82 8.2 | 10.8
#pragma once

#include <algorithm>
#include <cstdint>

namespace kq {
namespace rows {

constexpr uint32_t kThreads = 256;
constexpr uint32_t kSmem = 224 * 1024, kMost = 16;  // shared memory for the activations (of four rows at most); rows of a call

struct Call {
  bool i4;
  uint32_t n, k, m;
  uint32_t sm_count;
};
inline uint32_t per_step(const Call& c) { return c.i4 ? 32u : 16u; }               // weights of a 16-byte step
inline uint32_t rows_of_cta(const Call& c) { return c.m > 2 ? 4u : c.m; }
// Bytes of staged activations.
inline uint64_t staged_bytes(const Call& c) {
  return static_cast<uint64_t>((c.k / per_step(c)) | 1u) * (per_step(c) / 4u) * rows_of_cta(c) * 16u;
}
// Threads that share two channels, log2: as few as still give every SM the CTAs it holds (three at most), at least two steps
// each; fewer mean fewer reductions and fewer CTAs that stage the activations.
inline uint32_t lanes_log2(const Call& c) {
  const uint64_t fit = kSmem / (staged_bytes(c) + 1024u), pairs = (static_cast<uint64_t>(c.n) + 1u) / 2u;
  const uint64_t want = static_cast<uint64_t>(c.sm_count) * kThreads * (fit < 1 ? 1 : fit > 3 ? 3 : fit);
  uint32_t lanes = 2;
  while (lanes < 8 && (pairs << lanes) < want && (2u << lanes) * 2u <= c.k / per_step(c) + 1u) ++lanes;
  return lanes;
}

// This kernel: a launch and its trips to memory, what a thread multiplies one step after the other, the instructions of
// every weight (some of them for every activation row), and the activations that every CTA stages; int4 by waves of the two
// CTAs that a multiprocessor holds, half way between whole and part waves.
inline double estimate(const Call& c) {
  const uint32_t passes = (c.m + 3) / 4, lanes = 1u << lanes_log2(c), pairs = (c.n + 1) / 2;
  const double x = rows_of_cta(c), k = c.k, mega = static_cast<double>(c.n) * k * passes * 1e-6;
  const uint64_t ctas = (static_cast<uint64_t>(pairs) * lanes + kThreads - 1) / kThreads * passes;
  if (c.i4) {
    const uint64_t resident = std::min<uint64_t>(2, kSmem / (staged_bytes(c) + 1024u)), at_once = std::max<uint64_t>(1, c.sm_count * std::max<uint64_t>(1, resident));
    const double waves = ctas <= at_once ? 1.0 : 0.5 * ((ctas + at_once - 1) / at_once + static_cast<double>(ctas) / at_once);
    const double trips = 212 + (waves - 1.0) * std::min(212.0, 80 + k / 4);  // a wave's own; those of a short k overlap the next one's
    return 33 + 0.021 * x * k + trips + waves * (0.0198 * x * k + 0.352 * x * k * std::max<uint64_t>(1, resident) / lanes) + 14.6 * mega;
  }
  return 226 + 0.013 * x * k + mega * (0.7 + 7.6 * x) + 0.82 * x * k / lanes + static_cast<double>(ctas) / c.sm_count * (45 + 0.0123 * x * k);
}
// The generic kernel: a warp to a channel and four rows, one trip to memory after the other.
inline double estimate_generic(const Call& c) {
  const double trips = c.i4 ? (c.k + 255) / 256 : (c.k + 511) / 512, x = std::min(c.m, 4u), passes = (c.m + 3) / 4;
  const double all = c.n * passes * trips * 1e-3;
  return c.i4 ? 167 + trips * (18 + 18 * x) + all * (7.8 + 8.8 * x) : 149 + trips * (34 + 38 * x) + all * (37 + 12 * x);
}
constexpr double kNeighbour = 200;  // a norm or a residual add in a launch of its own
// The many-row kernel: its launches, and what kq_exact_geometry.h expects of its tiles.
inline double estimate_many_row(uint64_t clocks, bool binary16) { return (binary16 ? 106 : 275) + clocks * (95.6 / 1920); }

inline bool supports(const Call& c) {
  return c.m >= 1 && c.m <= kMost && c.n > 0 && c.k > 0 && c.k % per_step(c) == 0 && staged_bytes(c) <= kSmem;
}
// (a twentieth in favour of the others: of two that are level the one with fewer forms)
inline bool preferred(const Call& c, double other) { return estimate(c) * 1.05 <= other; }

}  // namespace rows
}  // namespace kq
