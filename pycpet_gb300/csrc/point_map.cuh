// point_map.cuh -- which points a thread of the grid kernels takes.
// Compiles as host C++ too.
#pragma once

#ifdef __CUDACC__
#define CPETGB_DEV __device__ __forceinline__
#else
#define CPETGB_DEV inline
#endif

namespace cpetgb {

// Which points a frame's threads take (u: thread of the frame, k: its k-th
// point): -1 for none.  stride: the lattice stride S, or 0.  A frame may have up to
// 2^31 - 1 points, so nothing here is rounded up past n_points in an int.
struct PointMap {
  int stride, lat_threads, lat_end, rest;  // columns x groups; rounded up to a warp; first other point
  int n_points;

  template <int PPT>
  CPETGB_DEV void set(int s, int P) {
    n_points = P;
    stride = s;
    const int groups = s > 0 ? P / s / PPT : 0;
    lat_threads = s * groups;
    lat_end = (lat_threads + 31) & ~31;
    rest = lat_threads * PPT;
  }
  // Threads of the frame that have points, rounded up to a warp.
  template <int PPT>
  CPETGB_DEV int threads() const {
    const int others = n_points - rest;
    return lat_end + (others > 0 ? (others - 1) / (32 * PPT) + 1 : 0) * 32;
  }
  CPETGB_DEV bool column(int u) const { return u < lat_end; }  // uniform across a warp
  template <int PPT>
  CPETGB_DEV int point(int u, int k) const {
    if (u < lat_end) {
      if (u >= lat_threads) return -1;
      const int g = u / stride;
      return (g * PPT + k) * stride + (u - g * stride);
    }
    const unsigned v = static_cast<unsigned>(u - lat_end);
    const unsigned off = (v >> 5) * (32u * PPT) + 32u * k + (v & 31u);
    return off < static_cast<unsigned>(n_points - rest) ? rest + static_cast<int>(off) : -1;
  }
};

}  // namespace cpetgb
