// Index arithmetic of the sampling kernels over a call's points, checked on the
// host by tests/cpp/point_index_test.cpp. A call has up to 2^31 - 1 points, so
// a point's coordinates lie beyond an int's range (3 t), and so does the first
// number past the last point that a grid-wide stride reaches: both are 64 bits.
#pragma once
#include "cell_index.h"

namespace birp {

using PointIndex = long long;

constexpr int kPointThreads = 256, kPointBlocks = 4096;

// CTAs of a call of n points (n >= 1)
BIRP_HD int point_blocks(int n) {
  const PointIndex b = ((PointIndex)n + kPointThreads - 1) / kPointThreads;
  return b < kPointBlocks ? (int)b : kPointBlocks;
}
// First point of thread `thread` of CTA `block`, and from each to its next.
BIRP_HD PointIndex points_first(unsigned block, unsigned threads, unsigned thread) {
  return (PointIndex)block * threads + thread;
}
BIRP_HD PointIndex points_step(unsigned blocks, unsigned threads) { return (PointIndex)blocks * threads; }
// Place of point t's x coordinate.
BIRP_HD PointIndex point_coords(PointIndex t) { return 3 * t; }

}  // namespace birp
