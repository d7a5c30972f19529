// Sums over a cluster of kCluster blocks of 256 threads, in a fixed order.
#pragma once
#include <cooperative_groups.h>

namespace sbe {

constexpr int kCluster = 8;

// |v|: sqrt(x^2 + y^2) where that neither overflows nor underflows, |x| for real values (FP64
// hypot costs about three times as much on the two-wide FP64 pipe)
__device__ __forceinline__ double cabs_d(double2 v) {
  const double a = fabs(v.x), b = fabs(v.y);
  if (b == 0.0) return a;
  const double m = fmax(a, b);
  if (m > 1e-140 && m < 1e140) return sqrt(fma(v.x, v.x, v.y * v.y));
  return hypot(v.x, v.y);
}

// Sums of the N values over the block (256 threads), returned to every thread.  An FP64
// instruction holds its scheduler for 64 clocks in every warp that issues it, so the warps that
// hold nothing (live false, the same over a warp) leave out the first sums and one warp per value
// forms the last ones.
template <int N>
__device__ __forceinline__ void block_sums(double (&v)[N], bool live) {
  __shared__ double red[N][8], tot[N];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (live) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int i = 0; i < N; ++i) v[i] += __shfl_down_sync(0xffffffffu, v[i], o);
  }
  __syncthreads();
  if (lane == 0)
#pragma unroll
    for (int i = 0; i < N; ++i) red[i][warp] = live ? v[i] : 0.0;
  __syncthreads();
  if (warp < N) {
    double x = lane < 8 ? red[warp][lane] : 0.0;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane == 0) tot[warp] = x;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = tot[i];
}

// ... and over the cluster (also a cluster barrier: what every block read before it may be
// overwritten after it); no block leaves before the others have read its sums
__device__ __forceinline__ void cluster_sum2(double& a, double& b, bool live) {
  namespace cg = cooperative_groups;
  __shared__ double part[2], all[2];
  cg::cluster_group cl = cg::this_cluster();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double v[2] = {a, b};
  block_sums(v, live);
  if (threadIdx.x == 0) {
    part[0] = v[0];
    part[1] = v[1];
  }
  cl.sync();
  if (warp < 2) {
    double x = lane < kCluster ? cl.map_shared_rank(part, lane)[warp] : 0.0;
#pragma unroll
    for (int o = 1; o < kCluster; o <<= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane == 0) all[warp] = x;
  }
  cl.sync();
  a = all[0];
  b = all[1];
}

}  // namespace sbe
