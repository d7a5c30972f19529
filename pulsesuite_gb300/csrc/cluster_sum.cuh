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

// sums of the N values over the block (256 threads), returned to every thread; a dependent
// FP64 addition takes about 130 clocks, so the values go together
template <int N>
__device__ __forceinline__ void block_sums(double (&v)[N]) {
  __shared__ double red[N][8];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] += __shfl_down_sync(0xffffffffu, v[i], o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int i = 0; i < N; ++i) red[i][threadIdx.x >> 5] = v[i];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const double* r = red[i];
    v[i] = ((r[0] + r[1]) + (r[2] + r[3])) + ((r[4] + r[5]) + (r[6] + r[7]));
  }
}

// ... and over the cluster (also a cluster barrier: what every block read before it may be
// overwritten after it); no block leaves before the others have read its sums
__device__ __forceinline__ void cluster_sum2(double& a, double& b) {
  namespace cg = cooperative_groups;
  __shared__ double part[2];
  cg::cluster_group cl = cg::this_cluster();
  double v[2] = {a, b};
  block_sums(v);
  if (threadIdx.x == 0) {
    part[0] = v[0];
    part[1] = v[1];
  }
  cl.sync();
  double p[2][kCluster];
#pragma unroll
  for (int r = 0; r < kCluster; ++r) {
    const double* q = cl.map_shared_rank(part, r);
    p[0][r] = q[0];
    p[1][r] = q[1];
  }
  auto sum = [](const double* x) {
    return ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));
  };
  a = sum(p[0]);
  b = sum(p[1]);
  cl.sync();
}

}  // namespace sbe
