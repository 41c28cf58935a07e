// Layer windows of the MUSCL/MFCT edges and work items of their mean-gradient
// layers (host and device, no CUDA header).
#pragma once
#ifdef __CUDACC__
#define FGB_HOST_DEVICE __host__ __device__ inline
#else
#define FGB_HOST_DEVICE inline
#endif

namespace fgb {

// The layers [first, end) (0-based) of an edge with hi layers that take the
// gradients of its up- and downwind triangles: those z (1-based) with
// gm0 <= z <= gm1 - 1, none if gm0 < 0. gm0 and gm1 come from the nodes' level
// tables, which a restart record supplies as they are: whatever they hold, the
// window stays within the edge's layers.
struct TriangleWindow {
  int first, end;
};
FGB_HOST_DEVICE TriangleWindow triangle_window(int gm0, int gm1, int hi) {
  auto below = [hi](int z) { return (z < 1 ? 1 : (z <= hi ? z : hi + 1)) - 1; };  // layers above layer z
  const int first = gm0 < 0 ? hi : below(gm0), end = gm0 < 0 ? hi : below(gm1);
  return TriangleWindow{first, end > first ? end : first};
}

// Work item of a thread of the mean-gradient kernel: two threads (one per node)
// for each of the kMeanRun layers of a run. The run's index is formed from the
// block's, so that it does not overflow for any list that int can count (a
// thread index over the whole grid wrapped at 2^28 runs).
constexpr int kMeanRun = 8;  // layers per run of DMesh::mean_seg
struct MeanItem {
  int run, layer, side;
};
FGB_HOST_DEVICE MeanItem mean_item(unsigned block, unsigned threads, unsigned thread) {
  return MeanItem{(int)(block * (threads / (2 * kMeanRun)) + thread / (2 * kMeanRun)), (int)(thread / 2 % kMeanRun),
                  (int)(thread & 1)};
}

}  // namespace fgb
