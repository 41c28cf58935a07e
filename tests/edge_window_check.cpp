// The layer windows of MUSCL/MFCT edges (fgb::triangle_window) against the condition they stand for: a layer z
// (1-based) of 1..hi takes the triangles' gradients if gm0 >= 0, z >= gm0 and z <= gm1 - 1. Prints the number of
// differences, over every small window, empty and inverted ones, starts above the surface and ends past the bottom,
// and over the mean-gradient kernel's items (fgb::mean_item) up to the longest list.
#include <climits>
#include <cstdio>
#include <initializer_list>

#include "fgb_window.hpp"

int main() {
  long long bad = 0;
  for (int hi = 0; hi <= 9; ++hi)
    for (int gm0 : {INT_MIN, -7, -1, 0, 1, 2, 3, 5, 8, 9, 10, 11, 40, INT_MAX})
      for (int gm1 : {INT_MIN, -7, -1, 0, 1, 2, 3, 4, 6, 9, 10, 11, 12, 40, INT_MAX}) {
        const fgb::TriangleWindow w = fgb::triangle_window(gm0, gm1, hi);
        if (w.first < 0 || w.end < w.first || w.end > hi) ++bad;
        for (int z = 1; z <= hi; ++z) {
          const bool in = gm0 >= 0 && z >= gm0 && (long long)z <= (long long)gm1 - 1;
          bad += in != (z - 1 >= w.first && z - 1 < w.end);
        }
      }
  // The mean-gradient kernel's items: consecutive runs over all blocks of the longest list (2^29 runs of an int count)
  for (unsigned block : {0u, 1u, 7u, (1u << 24) - 1, 1u << 24, (1u << 24) + 5, (1u << 25) - 1})
    for (unsigned thread = 0; thread < 256; ++thread) {
      const fgb::MeanItem it = fgb::mean_item(block, 256, thread);
      const long long item = (256LL * block + thread) / 2;
      bad += it.run != item / fgb::kMeanRun || it.layer != item % fgb::kMeanRun || it.side != (int)(thread & 1);
    }
  std::printf("%lld\n", bad);
  return bad != 0;
}
