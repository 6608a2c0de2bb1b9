// Host-side check of the line between the kernels for few rows over row-major weights (karume_b200/csrc/kq_rows_line.h and
// kq_exact_geometry.h): reads lines "int4? n k m binary16? other group" from standard input, with other 0 the generic kernel, 1 the
// many-row one, and prints 1 where the kernel for row-major weights is taken, on a device of 148 multiprocessors.
#include <cstdio>

#include "kq_exact_geometry.h"
#include "kq_rows_line.h"

int main() {
  const uint32_t slots[kq::exact::kMaxClusterSplits + 1] = {0, 74, 33, 0, 15};
  unsigned i4, n, k, m, half, other, group;
  while (std::scanf("%u %u %u %u %u %u %u", &i4, &n, &k, &m, &half, &other, &group) == 7) {
    const kq::rows::Call call = {i4 != 0, n, k, m, 148};
    const int math = half ? kq::exact::kHalf1 : kq::exact::kBf3;
    const uint64_t clocks = kq::exact::choose_geometry(m, n, (n + 255) / 256, kq::exact::steps_of(k, math, i4 ? group : 0, kq::exact::chain_of(math, !i4)), math,
                                                       !i4, true, slots, 256u << 20).clocks;
    const double theirs = other ? kq::rows::estimate_many_row(clocks, half != 0) : kq::rows::estimate_generic(call);
    std::printf("%d\n", kq::rows::supports(call) && kq::rows::preferred(call, theirs) ? 1 : 0);
  }
  return 0;
}
