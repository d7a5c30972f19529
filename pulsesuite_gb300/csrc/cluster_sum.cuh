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

// sums of a and b over the block, returned to every thread
__device__ __forceinline__ void block_sum2(double& a, double& b) {
  __shared__ double red[2][8];
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_down_sync(0xffffffffu, a, o);
    b += __shfl_down_sync(0xffffffffu, b, o);
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = a;
    red[1][threadIdx.x >> 5] = b;
  }
  __syncthreads();
  a = b = 0.0;
#pragma unroll
  for (int w = 0; w < 8; ++w) {
    a += red[0][w];
    b += red[1][w];
  }
}

// ... and over the cluster (also a cluster barrier: what every block read before it may be
// overwritten after it); no block leaves before the others have read its sums
__device__ __forceinline__ void cluster_sum2(double& a, double& b) {
  namespace cg = cooperative_groups;
  __shared__ double part[2];
  cg::cluster_group cl = cg::this_cluster();
  block_sum2(a, b);
  if (threadIdx.x == 0) {
    part[0] = a;
    part[1] = b;
  }
  cl.sync();
  a = b = 0.0;
  for (int r = 0; r < kCluster; ++r) {
    const double* q = cl.map_shared_rank(part, r);
    a += q[0];
    b += q[1];
  }
  cl.sync();
}

}  // namespace sbe
