// The spline solve in one launch.
//
// The FMM spline is a tridiagonal solve: pivots p_i = 2 (d_{i-1} + d_i) - d_{i-1}^2 / p_{i-1},
// a forward sweep c_i -= t_i c_{i-1} with t_i = d_{i-1} / p_{i-1}, a backward sweep
// c_i = (c_i - d_i c_{i+1}) / p_i.  On ascending knots whose adjacent spacings differ by at
// most a factor 1 / rho, t_i and d_i / p_i are at most 1 / (2 + 1.5 rho) (0.286 on a uniform
// grid), so each recurrence forgets its start: a thread takes kSeg points after a warm-up
// started from zero, long enough for 2^-64 (36 points on a uniform grid, 64 at most; the pivots,
// which contract by t^2, half of that).  The first and last segments start from the exact
// ends.  FP64 issues two operations per clock and SM and a dependent FMA takes about 130
// clocks, so the chains are what costs: real and imaginary parts have threads of their own,
// the pivots come from the determinants theta_i = b_i theta_{i-1} - d_{i-1}^2 theta_{i-2} (one
// dependent FMA a point, p_i = theta_i / theta_{i-1} beside it), and a block holds few points
// (64, all fields of one set of knots) so that the grid spreads them over the SMs.
// A value that is not finite reaches the coefficients of some 100 points only; a solve from end to
// end spreads it over all, which the calls that resample one wire keep (bad, k_spline_eval).
// Mean of the solves of a step (4 fields on 4096 points, 5 on Nr = 230): 17.5 ms with one thread
// per field, 32 us with the chains in threads of their own, 22 us with the pivots' coefficients and
// reciprocals formed by all threads (3 fields on 8192, 5 on 514: 31 -> 22 us).
#include "spline.cuh"
#include "fp_bits.cuh"

namespace sbe {
namespace {

constexpr int kTile = kSplTile, kSeg = 8, kWarm = 64, kWarmP = 32, kFields = 5;
constexpr int kCap = kTile + 2 * kWarm + kWarmP + 16;   // points a block holds
constexpr int kThreads = 256;

// complex over real as NumPy divides by (d + 0i)
__device__ __forceinline__ double2 cdivr(double2 a, double d) { return cscale(a, 1.0 / d); }

__global__ void __launch_bounds__(kThreads) k_spline(SplBatch s) {
  pdl_enter();
  __shared__ int bad;
  __shared__ double2 c1[kFields][kCap], c2[kFields][kCap];
  __shared__ double x[kCap], ip[kCap], id[kCap], tt[kCap], mm[kCap];
  __shared__ double red[2][kThreads / 32];
  const int g = blockIdx.y, tid = threadIdx.x, nf = s.nf;
  if (tid == 0) bad = 0;
  int n = s.n0;
  long long ko = 0;
  if (s.off) {
    n = s.n[g * nf];
    ko = s.off[2 * g * nf];
  }
  auto voff = [&](int f) {
    return s.off ? s.off[2 * (g * nf + f) + 1] : (long long)(g * nf + f) * s.n0;
  };
  const int s0 = blockIdx.x * kTile;
  if (s0 >= n) return;
  const int e = min(s0 + kTile, n), sb = max(0, s0 - 1);   // sb: first point the sweeps keep
  const double* gx = s.X + ko;
  const int x0 = max(0, sb - kWarm - 1 - kWarmP - 1), xe = min(n, e + kWarm + 1);
  for (int i = x0 + tid; i < xe; i += kThreads) x[i - x0] = gx[i];
  __syncthreads();
  // spacings: their range over the block's points sets the warm-up
  double lo = INFINITY, hi = 0.0;
  for (int i = x0 + tid; i < xe - 1; i += kThreads) {
    const double d = x[i - x0 + 1] - x[i - x0];
    id[i - x0] = rcp64(d);
    lo = fmin(lo, fabs(d));
    hi = fmax(hi, fabs(d));
  }
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if ((tid & 31) == 0) {
    red[0][tid >> 5] = lo;
    red[1][tid >> 5] = hi;
  }
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) {
    lo = fmin(lo, red[0][w]);
    hi = fmax(hi, red[1][w]);
  }
  // 64 ln 2 / ln(2 + 1.5 rho), one point of margin
  const float rho = (float)(lo / hi);
  const int warm = rho > 0.f ? min(kWarm, (int)(44.37f / __logf(2.f + 1.5f * rho)) + 2) : kWarm;
  const double is = rcp64(hi);
  const bool det = rho > 1e-4f;   // the determinants of 40 points stay in range
  const int fe = min(n, e + warm);                // forward sweep up to here
  const int l0 = max(0, sb - warm - 1);           // first right-hand side
  // reciprocal pivots over [l0, fe), with t_{i+1} and d_i / p_i
  if (det) {
    double *bb = reinterpret_cast<double*>(c1[0]), *th = reinterpret_cast<double*>(c1[1]);
    // b_i and d_{i-1}^2 (in mm), spacings in units of hi: a warp's FP64 instruction holds its
    // scheduler for 64 clocks however few its lanes, so only the recurrence itself stays with
    // the few threads of the segments
    for (int i = max(0, l0 - warm / 2) + tid; i < fe; i += kThreads) {
      const int j = i - x0;
      const double dm = i > 0 ? (x[j] - x[j - 1]) * is : 0.0;
      const double dp = i < n - 1 ? (x[j + 1] - x[j]) * is : 0.0;
      bb[j] = i == 0 ? -dp : i == n - 1 ? -dm : 2.0 * (dm + dp);
      mm[j] = -(dm * dm);
    }
    __syncthreads();
    for (int a = l0 + tid * kSeg; a < fe; a += kThreads * kSeg) {
      const int b = min(a + kSeg, fe);
      double t1 = 1.0, t2 = 0.0;   // theta_{i-1}, theta_{i-2}
#pragma unroll 4
      for (int i = max(0, a - warm / 2); i < b; ++i) {
        const int j = i - x0;
        const double t0 = fma(bb[j], t1, mm[j] * t2);
        if (i >= a) {
          ip[j] = t1;
          th[j] = t0;
        }
        t2 = t1;
        t1 = t0;
      }
    }
    __syncthreads();
    for (int i = l0 + tid; i < fe; i += kThreads) {
      const int j = i - x0;
      const double dp = i < n - 1 ? (x[j + 1] - x[j]) * is : 0.0;
      const double r = ip[j] * rcp64(th[j]);   // hi / p_i
      ip[j] = r * is;
      mm[j] = tt[j + 1] = dp * r;
    }
  } else {
    for (int a = l0 + tid * kSeg; a < fe; a += kThreads * kSeg) {
      const int b = min(a + kSeg, fe);
      double r = 0.0;   // 1 / p of the point before
      for (int i = max(0, a - kWarmP); i < b; ++i) {
        const int j = i - x0;
        const double dp = i < n - 1 ? x[j + 1] - x[j] : 0.0;
        const double dm = i > 0 ? x[j] - x[j - 1] : 0.0;
        const double bi = i == 0 ? -dp : i == n - 1 ? -dm : 2.0 * (dm + dp);
        r = rcp64(bi - dm * dm * r);
        if (i >= a) {
          ip[j] = r;
          mm[j] = tt[j + 1] = dp * r;
        }
      }
    }
  }
  // (y_{i+1} - y_i) / d_i, held in c2 until the sweeps
  for (int f = 0; f < nf; ++f) {
    const double2* gy = s.Y + voff(f);
    for (int i = max(0, l0 - 1) + tid; i < min(fe, n - 1); i += kThreads)
      c2[f][i - x0] = cscale(csub(gy[i + 1], gy[i]), id[i - x0]);
  }
  __syncthreads();
  // right-hand side: second differences and the FMM end conditions
  const int nl = fe - l0;
  for (int q = tid; q < nf * nl; q += kThreads) {
    const int f = q / nl, i = l0 + q % nl, j = i - x0;
    const double2* dl = c2[f] + j;
    double2 c;
    if (i >= 1 && i <= n - 2) {
      c = csub(dl[0], dl[-1]);
    } else if (i == 0) {
      c = csub(cdivr(csub(dl[2], dl[1]), x[3] - x[1]), cdivr(csub(dl[1], dl[0]), x[2] - x[0]));
      const double d0 = x[1] - x[0];
      c = cdivr(cscale(c, d0 * d0), x[3] - x[0]);
    } else {
      c = csub(cdivr(csub(dl[-1], dl[-2]), x[j] - x[j - 2]),
               cdivr(csub(dl[-2], dl[-3]), x[j - 1] - x[j - 3]));
      const double dn = x[j] - x[j - 1];
      c = cdivr(cscale(make_double2(-c.x, -c.y), dn * dn), x[j] - x[j - 3]);
    }
    c1[f][j] = c;
  }
  __syncthreads();
  // forward sweep over [sb, fe): one (field, component, segment) per thread
  {
    const int ns = (fe - sb + kSeg - 1) / kSeg;
    for (int q = tid; q < 2 * nf * ns; q += kThreads) {
      const int f = q / ns, a = sb + (q % ns) * kSeg, b = min(a + kSeg, fe);
      const double* u = reinterpret_cast<const double*>(c1[f >> 1]) + (f & 1);
      double* w = reinterpret_cast<double*>(c2[f >> 1]) + (f & 1);
      int i = max(1, a - warm);
      double v = i == 1 ? u[0] : 0.0;   // i == 1: x0 = 0
      if (a == 0) w[0] = u[0];
#pragma unroll 4
      for (; i < b; ++i) {
        const int j = i - x0;
        v = fma(-tt[j], v, u[2 * j]);
        if (i >= a) w[2 * j] = v;
      }
    }
  }
  __syncthreads();
  // c_i / p_i, so that the backward sweep is one FMA per component
  for (int q = tid; q < nf * (fe - sb); q += kThreads) {
    const int f = q / (fe - sb), j = sb + q % (fe - sb) - x0;
    c2[f][j] = cscale(c2[f][j], ip[j]);
  }
  __syncthreads();
  // backward sweep over [sb, e], result in c1
  {
    const int e1 = min(e + 1, n), ns = (e1 - sb + kSeg - 1) / kSeg;
    for (int q = tid; q < 2 * nf * ns; q += kThreads) {
      const int f = q / ns, a = sb + (q % ns) * kSeg, b = min(a + kSeg, e1);
      const double* u = reinterpret_cast<const double*>(c2[f >> 1]) + (f & 1);
      double* w = reinterpret_cast<double*>(c1[f >> 1]) + (f & 1);
      int i = min(n - 2, min(b - 1 + warm, fe - 1));
      double v = 0.0;
      if (fe == n && i == n - 2) v = u[2 * (n - 1 - x0)];   // the exact end
      if (b == n) w[2 * (n - 1 - x0)] = v;
#pragma unroll 4
      for (; i >= a; --i) {
        const int j = i - x0;
        v = fma(-mm[j], v, u[2 * j]);
        if (i < b) w[2 * j] = v;
      }
    }
  }
  __syncthreads();
  // coefficients (spliner.py:1384-1394)
  for (int q = tid; q < nf * (e - s0); q += kThreads) {
    const int f = q / (e - s0), i = s0 + q % (e - s0), j = i - x0;
    const long long vo = voff(f);
    const double2* gy = s.Y + vo;
    double2 *gb = s.coef + 3 * vo, *gc = gb + n, *gd = gb + 2 * n;
    const double2 c = c1[f][j];
    if (not_finite(c.x)) atomicOr(&bad, 1 << 2 * f);
    if (not_finite(c.y)) atomicOr(&bad, 2 << 2 * f);
    gc[i] = cscale(c, 3.0);
    if (i < n - 1) {
      const double2 cn = c1[f][j + 1];
      gb[i] = csub(cscale(csub(gy[i + 1], gy[i]), id[j]),
                   cscale(cadd(cn, cscale(c, 2.0)), x[j + 1] - x[j]));
      gd[i] = cscale(csub(cn, c), id[j]);
    } else {
      const double2 cp = c1[f][j - 1];
      gb[i] = cadd(cscale(csub(gy[i], gy[i - 1]), id[j - 1]),
                   cscale(cadd(cp, cscale(c, 2.0)), x[j] - x[j - 1]));
      gd[i] = cscale(csub(c, cp), id[j - 1]);
    }
  }
  if (s.bad) {
    __syncthreads();
    if (tid == 0) s.bad[g * gridDim.x + blockIdx.x] = bad;
  }
}

}  // namespace

void launch_splines(const SplBatch& b, int ngroups, int nmax, cudaStream_t s) {
  launch(k_spline, dim3((nmax + kTile - 1) / kTile, ngroups), kThreads, 0, s, b);
}

}  // namespace sbe
