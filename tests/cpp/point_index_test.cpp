// Host check of the sampling kernels' index arithmetic
// (birp_cpp_gb300/csrc/point_index.h) at the smallest and largest calls: every
// thread's points run upwards, end, stay below n and have their coordinates in
// [0, 3 n), and together they are each of the n points once. Exit code = number
// of failures.
#include <climits>
#include <cstdio>
#include <vector>

#include "../../birp_cpp_gb300/csrc/point_index.h"

using namespace birp;

int main() {
  int fails = 0;
  for (int n : {1, 31, 32, 33, 255, 256, 257, 1048575, 1048576, 1048577, 715827882, 715827883, 2146435072, INT_MAX - 256,
                INT_MAX - 1, INT_MAX}) {
    const int blocks = point_blocks(n);
    if (blocks < 1 || blocks > kPointBlocks) {
      ++fails;
      continue;
    }
    const auto step = points_step(blocks, kPointThreads);
    // the first, a middle and the last CTAs, whole warps (first lane) and each lane
    for (int b : {0, blocks / 2, blocks - 1})
      for (int t : {0, 1, 31, 32, 224, 255}) {
        auto w = points_first(b, kPointThreads, t);
        long long passes = 0;
        for (; w < n && passes <= 2050; w += step, ++passes) {
          const auto c = point_coords(w);
          if (w < 0 || c < 0 || c + 2 >= 3ll * n) {
            ++fails;
            break;
          }
        }
        if (w < n) ++fails;  // went on past the last point
        if (passes != ((long long)n - ((long long)b * kPointThreads + t) + step - 1) / step &&
            (long long)b * kPointThreads + t < n)
          ++fails;
      }
    if (n <= 1048577) {
      std::vector<int> seen(n, 0);
      for (int b = 0; b < blocks; ++b)
        for (int t = 0; t < kPointThreads; ++t)
          for (auto w = points_first(b, kPointThreads, t); w < n; w += step) ++seen[w];
      for (int s : seen) fails += s != 1;
    }
  }
  std::printf("%d failures\n", fails);
  return fails != 0;
}
