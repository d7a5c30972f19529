// Forsythe-Malcolm-Moler cubic splines (spliner.py:1329-1394) of complex values, a batch of
// problems per launch: nf consecutive problems share their knots.
#pragma once
#include <cuda_runtime.h>

#include "sbe_internal.cuh"

namespace sbe {

struct SplBatch {
  const double* X;      // knots base
  const double2* Y;     // values base
  double2* coef;        // 3 per value: b, c, d blocks of n
  const int* n;         // knots per problem (nullptr: n0 for all)
  const long long* off; // per problem: knot and value offset (nullptr: 0 and p * n0)
  int n0, nf;           // nf: 1 to 5
  int* bad;             // per group and tile (or null): bits 2 f, 2 f + 1 of field f's real and
                        // imaginary part with a coefficient that is not finite
};

// every problem needs at least kSplMin knots
constexpr int kSplMin = 4;
// points whose coefficients one block stores, and the tiles of n knots
constexpr int kSplTile = 64;
__host__ __device__ constexpr int spl_tiles(int n) { return (n + kSplTile - 1) / kSplTile; }
// complex values that hold the tiles' words of n knots
__host__ __device__ constexpr int spl_bad_elems(int n) { return (spl_tiles(n) + 3) / 4; }
void launch_splines(const SplBatch& b, int ngroups, int nmax, cudaStream_t s);

// spliner.py:1137-1167 locate on ascending knots
__device__ __forceinline__ int locate_sorted(const double* xx, int n, double x) {
  if (x < xx[0]) return 0;
  if (x >= xx[n - 1]) return n - 1;
  int jl = 0, ju = n;
  while (ju - jl > 1) {
    const int jm = (ju + jl) >> 1;
    if (x >= xx[jm])
      jl = jm;
    else
      ju = jm;
  }
  return jl;
}

__device__ __forceinline__ double2 spl_eval(const double2* y, const double2* b, int n, int i,
                                            double dx) {
  const double2* c = b + n;
  const double2* d = b + 2 * n;
  double2 t = cadd(c[i], cscale(d[i], dx));
  t = cadd(b[i], cscale(t, dx));
  return cadd(y[i], cscale(t, dx));
}

}  // namespace sbe
