// 3-D PSTD field step: six field components on an nx x ny x nz grid (C order, z
// fastest), spectral curls by 3-D FFTs built from three axis passes, the k-space
// curl multiply fused into the x pass and the field update fused into the last
// (inverse z) pass.
//
// The reference has no 3-D Maxwell stepper either (its 3-D driver sets E
// analytically, sbetestpropnov30.py:709); the pieces are the q-space derivative
// f (i q) along each axis (PSTD3D/usefulsubs.py:233-380), the grids of
// typespace.py:815-849 and helpers.py:838-863, the absorbing mask multiply of
// ApplyABC (usefulsubs.py:584-609) and the longitudinal field of ElongfromRho
// (rhoPJ.py:703-880).  Leapfrog:
//   H^{n+1/2} = H^{n-1/2} - dt/mu0 curl E^n,
//   E^{n+1}   = mask (E^n + dt/eps (curl H^{n+1/2} - J)).
//
// One curl of a field triple F (3 x c128 N, N = nx ny nz) runs five passes:
//   1  z lines, forward (FP64 field -> work W)
//   2  y lines, forward (in place)
//   3  x lines: forward, c = i q x F at every (kx, ky, kz), inverse (in place; a block
//      holds the x lines of all three components of its (ky, kz) columns)
//   4  y lines, inverse
//   5  z lines, inverse, 1/N, and out += a c (+ ja J), mask (FP64 out)
// Every transform is a Stockham sequence in shared memory (FP64 in radix 4).  The work array
// W is FP64 or FP32 complex (chosen at creation): with FP32 work the three middle
// passes move half the bytes and the FP64 field is touched only by passes 1 and 5.
#include <algorithm>
#include <cmath>
#include <vector>

#include "fft64.cuh"
#include "fp_bits.cuh"
#include "pstd3d.cuh"

namespace sbe {
namespace {

constexpr double kMu0 = 1.25663706127e-6;   // CODATA 2022 (scipy.constants.mu_0)
constexpr int kThreads = 256;
constexpr int kSmemMax = 200 * 1024;

template <typename T>
__device__ __forceinline__ T mk(double a, double b);
template <>
__device__ __forceinline__ double2 mk<double2>(double a, double b) {
  return make_double2(a, b);
}
template <>
__device__ __forceinline__ float2 mk<float2>(double a, double b) {
  return make_float2((float)a, (float)b);
}

template <typename T>
__device__ __forceinline__ T tmul(T a, T b) {
  T r;
  r.x = a.x * b.x - a.y * b.y;
  r.y = a.x * b.y + a.y * b.x;
  return r;
}

template <typename T>
__device__ __forceinline__ T twd(const double2* tw, const float2* twf, int i);
template <>
__device__ __forceinline__ double2 twd<double2>(const double2* tw, const float2*, int i) {
  return __ldg(&tw[i]);
}
template <>
__device__ __forceinline__ float2 twd<float2>(const double2*, const float2* twf, int i) {
  return __ldg(&twf[i]);
}

// Radix-2 Stockham over shared memory: ntr = 2^lgtr transforms of length L = 2^lg,
// element p of transform c at a[p * ps + c * cs]; consecutive threads walk c
// (c_fast) or p.  dir -1: exp(-i ...), +1: exp(+i ...).  Returns the buffer
// holding the result in natural order.
template <typename T>
__device__ T* fft_smem(T* a, T* b, int lg, int lgtr, int ps, int cs, bool c_fast, int dir,
                       const double2* tw, const float2* twf) {
  const int L = 1 << lg;
  const int half = L >> 1;
  const int total = half << lgtr;
  for (int ns = 1; ns < L; ns <<= 1) {
    const int tws = L / (2 * ns);
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
      int j, c;
      if (c_fast) {
        c = idx & ((1 << lgtr) - 1);
        j = idx >> lgtr;
      } else {
        j = idx & (half - 1);
        c = idx >> (lg - 1);
      }
      const int k = j & (ns - 1);
      const T u = a[j * ps + c * cs];
      T v = a[(j + half) * ps + c * cs];
      T w = twd<T>(tw, twf, k * tws);
      if (dir > 0) w.y = -w.y;
      v = tmul(v, w);
      const int o = ((j - k) << 1) + k;
      T s0, s1;
      s0.x = u.x + v.x;
      s0.y = u.y + v.y;
      s1.x = u.x - v.x;
      s1.y = u.y - v.y;
      b[o * ps + c * cs] = s0;
      b[(o + ns) * ps + c * cs] = s1;
    }
    __syncthreads();
    T* t = a;
    a = b;
    b = t;
  }
  return a;
}

// The FP64 transforms run in radix 4 (fft64.cuh).
template <>
__device__ double2* fft_smem<double2>(double2* a, double2* b, int lg, int lgtr, int ps, int cs,
                                      bool c_fast, int dir, const double2* tw, const float2*) {
  return fft64(a, b, lg, lgtr, ps, cs, c_fast, dir, tw);
}

__host__ __device__ inline int ilog2i(int v) {
  int l = 0;
  while ((1 << l) < v) ++l;
  return l;
}

// Geometry of one pass: lines of length n along an axis of stride s (elements);
// lines are enumerated by (outer o, inner i), element p of line (o, i) at
// o * n * s + p * s + i (field f at f * N).
struct Pass {
  int n, lg, s, inner, tl, lgtl, nf;
  long long N;
  int dir;
  const double2* tw;
  const float2* twf;
};

// Generic line pass: nf fields.  Loads TL lines of each field (consecutive inner
// indices, or consecutive whole lines when s == 1), transforms them, stores them.
// in64 / out64: FP64 fields (pass 1 reads one, pass 5 writes one through the update
// epilogue); otherwise the work array (T) is read and written in place.
struct Upd {
  double2* out;            // FP64 destination (nullptr: store to work)
  const double2* J;        // optional current (FP64, 3 fields)
  double a, ja;            // out += a * result / N - ja * J
  const double* m0;        // masks per axis (nullptr: none)
  const double* m1;
  const double* m2;
  int nx, ny, nz;
  int store;               // 1: out = result / N (no update)
  float af[2], jf[2];      // the plane path's a / N and ja as FP32 pairs (hi, lo)
  int nabc[3];             // absorbing widths: the mask is exactly 1 further inside
};

template <typename T>
__global__ void __launch_bounds__(kThreads) k_line_pass(Pass P, const double2* in64, T* W,
                                                        Upd U) {
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smraw[];
  T* sa = reinterpret_cast<T*>(smraw);
  const int tl = P.tl, n = P.n;
  const int f = blockIdx.y;   // field
  T* sb = sa + (size_t)n * tl;
  // line block: lines (o, i0 .. i0 + tl - 1), or tl whole lines when s == 1
  long long base;
  if (P.s == 1) {
    base = (long long)blockIdx.x * tl * n;    // lines contiguous, element (c, p) at c n + p
  } else {
    const int bpo = P.inner / tl;             // blocks per outer index
    const int o = blockIdx.x / bpo, i0 = (blockIdx.x % bpo) * tl;
    base = (long long)o * n * P.s + i0;
  }
  const long long fo = (long long)f * P.N;
  const int total = n * tl;
  // smem layout: element p of line c at p * tl + c (strided) or c * n + p (s == 1)
  for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
    long long g;
    int sm;
    if (P.s == 1) {
      g = base + idx;                          // c = idx / n, p = idx % n
      sm = idx;
    } else {
      const int c = idx % tl, p = idx / tl;
      g = base + (long long)p * P.s + c;
      sm = p * tl + c;
    }
    T v;
    if (in64) {
      const double2 d = in64[fo + g];
      v = mk<T>(d.x, d.y);
    } else {
      v = W[fo + g];
    }
    sa[sm] = v;
  }
  __syncthreads();
  T* r;
  if (P.s == 1)
    r = fft_smem(sa, sb, P.lg, P.lgtl, 1, n, false, P.dir, P.tw, P.twf);
  else
    r = fft_smem(sa, sb, P.lg, P.lgtl, tl, 1, true, P.dir, P.tw, P.twf);
  const double invN = 1.0 / (double)((long long)U.nx * U.ny * U.nz);
  for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
    long long g;
    int sm;
    if (P.s == 1) {
      g = base + idx;
      sm = idx;
    } else {
      const int c = idx % tl, p = idx / tl;
      g = base + (long long)p * P.s + c;
      sm = p * tl + c;
    }
    const T v = r[sm];
    if (!U.out) {
      W[fo + g] = v;
      continue;
    }
    double vx = (double)v.x * invN, vy = (double)v.y * invN;
    double2 o;
    if (U.store) {
      o = make_double2(vx, vy);
    } else {
      o = U.out[fo + g];
      o.x += U.a * vx;
      o.y += U.a * vy;
      if (U.J) {
        const double2 j = U.J[fo + g];
        o.x -= U.ja * j.x;
        o.y -= U.ja * j.y;
      }
    }
    if (U.m0) {
      const long long yz = (long long)U.ny * U.nz;
      const int i = (int)(g / yz), jj = (int)((g / U.nz) % U.ny), k = (int)(g % U.nz);
      const double m = U.m0[i] * U.m1[jj] * U.m2[k];
      o.x *= m;
      o.y *= m;
    }
    U.out[fo + g] = o;
  }
}

// The x pass of the curl: a block holds the x lines of the three components of tl
// consecutive (y, z) columns; forward FFT, c = i q x F, inverse FFT, in place.
template <typename T>
__global__ void __launch_bounds__(kThreads) k_x_curl(Pass P, T* W, const double* qy,
                                                     const double* qz, const double* qx, int nz) {
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smraw[];
  T* sa = reinterpret_cast<T*>(smraw);
  const int tl = P.tl, n = P.n;
  T* sb = sa + (size_t)3 * n * tl;
  const int b0 = blockIdx.x * tl;             // first (y, z) column
  const int total = 3 * n * tl;               // element (f, p, c) at (f * n + p) * tl + c
  for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
    const int c = idx % tl, fp = idx / tl, p = fp % n, f = fp / n;
    sa[idx] = W[(long long)f * P.N + (long long)p * P.s + b0 + c];
  }
  __syncthreads();
  // 3 tl transforms: transform index t = f * tl + c, element p at (f n + p) tl + c =
  // p tl + (f n tl + c): not a single stride, so transform each component in turn
  T* r[3];
  for (int f = 0; f < 3; ++f)
    r[f] = fft_smem(sa + (size_t)f * n * tl, sb + (size_t)f * n * tl, P.lg, P.lgtl, tl, 1, true,
                    -1, P.tw, P.twf);
  // the curl at every (kx, column)
  for (int idx = threadIdx.x; idx < n * tl; idx += blockDim.x) {
    const int c = idx % tl, p = idx / tl;
    const int col = b0 + c;
    const double kx = qx[p], ky = qy[col / nz], kz = qz[col % nz];
    const T fx = r[0][idx], fy = r[1][idx], fz = r[2][idx];
    // i (k x F)
    const double cxr = ky * fz.x - kz * fy.x, cxi = ky * fz.y - kz * fy.y;
    const double cyr = kz * fx.x - kx * fz.x, cyi = kz * fx.y - kx * fz.y;
    const double czr = kx * fy.x - ky * fx.x, czi = kx * fy.y - ky * fx.y;
    r[0][idx] = mk<T>(-cxi, cxr);
    r[1][idx] = mk<T>(-cyi, cyr);
    r[2][idx] = mk<T>(-czi, czr);
  }
  __syncthreads();
  T* o[3];
  for (int f = 0; f < 3; ++f) {
    T* other = (r[f] == sa + (size_t)f * n * tl) ? sb + (size_t)f * n * tl : sa + (size_t)f * n * tl;
    o[f] = fft_smem(r[f], other, P.lg, P.lgtl, tl, 1, true, +1, P.tw, P.twf);
  }
  for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
    const int c = idx % tl, fp = idx / tl, p = fp % n, f = fp / n;
    W[(long long)f * P.N + (long long)p * P.s + b0 + c] = o[f][p * tl + c];
  }
}

// ElongfromRho in k space (rhoPJ.py:836-866) on the transformed fields
// S = [rho, Px, Py, Pz]: writes the ten spectra [E_PRho x, y, z, E_P x, y, z,
// E_Rho x, y, z, rho_B] into O.  small = (qx[1] - qx[0]) / 1e4 (:779).
__global__ void k_elong3(long long N, int ny, int nz, const double2* S, double2* O,
                         const double* qx, const double* qy, const double* qz, double small,
                         double inv_eps) {
  const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (g >= N) return;
  const long long yz = (long long)ny * nz;
  const double kx = qx[g / yz], ky = qy[(g / nz) % ny], kz = qz[g % nz];
  const double2 rk = S[g], px = S[N + g], py = S[2 * N + g], pz = S[3 * N + g];
  const double qs = kx * kx + ky * ky + kz * kz + small;
  const double2 qp = make_double2(kx * px.x + ky * py.x + kz * pz.x, kx * px.y + ky * py.y + kz * pz.y);
  // rho_term = -i rho inv_eps / qs ; P_term = -(q.P) inv_eps / qs
  const double2 rt = make_double2(rk.y * inv_eps / qs, -rk.x * inv_eps / qs);
  const double2 pt = make_double2(-qp.x * inv_eps / qs, -qp.y * inv_eps / qs);
  const double q3[3] = {kx, ky, kz};
  for (int c = 0; c < 3; ++c) {
    O[(long long)c * N + g] = make_double2((rt.x + pt.x) * q3[c], (rt.y + pt.y) * q3[c]);
    O[(long long)(3 + c) * N + g] = make_double2(pt.x * q3[c], pt.y * q3[c]);
    O[(long long)(6 + c) * N + g] = make_double2(rt.x * q3[c], rt.y * q3[c]);
  }
  O[9 * N + g] = make_double2(qp.y, -qp.x);   // rho_B = -i q.P
}

__global__ void k_tables3(int n, double d, double* x, double* q, double2* tw, float2* twf,
                          float2* qb, double* mask, int n_abc, double strength) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  {
    // the wavenumber of bit-reversed position j as an FP32 pair (the plane path's
    // spectrum order)
    int lg = 0;
    while ((1 << lg) < n) ++lg;
    const int jb = (int)(__brev((unsigned)j) >> (32 - lg));
    const double qv = (jb <= n / 2 ? jb : jb - n) * (2.0 * kPi / (n * d));
    const float hi = (float)qv;
    qb[j] = make_float2(hi, (float)(qv - (double)hi));
  }
  // GetSpaceArray: numpy linspace(-L/2, L/2, n) with L = (n - 1) d (typespace.py:815-849):
  // j * step + start, rounded as numpy does (no fused multiply-add), the last point = stop
  const double L = (n - 1) * d;
  const double start = -L / 2, stop = L / 2;
  const double step = (stop - start) / (double)(n - 1);
  x[j] = (j == n - 1) ? stop : __dadd_rn(__dmul_rn((double)j, step), start);
  const double dq = 2.0 * kPi / (n * d);
  q[j] = (j <= n / 2 ? j : j - n) * dq;
  double s, c;
  sincospi(-2.0 * (double)j / (double)n, &s, &c);
  tw[j] = make_double2(c, s);
  twf[j] = make_float2((float)c, (float)s);
  const int dd = j < n - 1 - j ? j : n - 1 - j;
  double m = 1.0;
  if (n_abc > 0 && dd < n_abc) {
    const double u = (double)(n_abc - dd) / n_abc;
    m = exp(-strength * u * u);
  }
  mask[j] = m;
}

// ---- FP32 work with (y, z) planes in shared memory: three passes per curl ------
// When a (y, z) plane of FP32 complex values fits in one block's shared memory
// (ny nz <= kPlaneMax) a curl is three passes instead of five:
//   A  per (x, component) plane: FP64 field -> FP32, forward transforms along z and y
//   B  x lines of tl (y, z) columns of all three components: forward along x, the curl
//      i q x F, inverse along x
//   C  per plane: inverse along y and z, out (+)= a curl / N (- ja J), mask; in the
//      field step C of the H update continues with pass A of the E update on the new
//      H it has just written (the elements are still in registers)
// The transforms are radix-2 decimation in frequency (natural order in, bit-reversed
// order out, exp(-i ...)) and its exact inverse, decimation in time (bit-reversed in,
// natural out, unnormalised).  The spectrum is never reordered: the curl is pointwise
// in k space and reads the wavenumber of position p as q[bitrev(p)].
//
// A thread takes up to four radix-2 stages of 16 elements in registers, so a line of
// 128 or 256 goes through shared memory once between its two groups of stages instead
// of before and after every pair of them, and the first and last group of a pass work
// straight from and to global memory.  The radix-4 sweeps over shared memory that this
// replaces bound all three passes (one plane per SM, 9 round trips of 128 KB forward):
// 256 x 128 x 128 step 1.14 -> 0.77 ms (per launch: A 157 -> 95 us, B 155 -> 81, C 339 -> 256;
// 2.7 TB/s in A and C, whose single block per SM alternates between memory and transforms;
// 1024 threads with groups of at most 8 elements 0.82 ms).
constexpr int kPlaneMax = 16384;   // FP32 complex elements of one plane (128 KB)
constexpr int kPlaneThreads = 512;
constexpr int kXThreads = 256;
constexpr int kXSmem = 96 * 1024;  // shared memory of one x-pass block's lines

// Complex arithmetic with one fixed rounding per product wherever the compiler puts it, on the
// two-wide FP32 instructions.
__device__ __forceinline__ float2 c_mul(float2 a, float2 w) {
  return __ffma2_rn(a, make_float2(w.x, w.x), make_float2(-__fmul_rn(a.y, w.y), __fmul_rn(a.x, w.y)));
}
__device__ __forceinline__ float2 c_mul2(float2 a, float2 w) {   // the imaginary sum turned round
  return make_float2(__fmaf_rn(a.x, w.x, -__fmul_rn(a.y, w.y)),
                     __fmaf_rn(a.x, w.y, __fmul_rn(a.y, w.x)));
}
__device__ __forceinline__ float2 c_mulc(float2 a, float2 w) {   // a conj(w)
  return __ffma2_rn(a, make_float2(w.x, w.x), make_float2(__fmul_rn(a.y, w.y), -__fmul_rn(a.x, w.y)));
}
__device__ __forceinline__ float2 c_add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 c_sub(float2 a, float2 b) {
  return __ffma2_rn(b, make_float2(-1.f, -1.f), a);
}

// Two radix-2 stages on x[0], x[ST], x[2 ST], x[3 ST] (positions m apart).
template <bool INV, int ST>
__device__ __forceinline__ void pair_stage(float2* x, float2 w1a, float2 w1b, float2 w2) {
  const float2 x0 = x[0], x1 = x[ST], x2 = x[2 * ST], x3 = x[3 * ST];
  if (!INV) {
    const float2 a0 = c_add(x0, x2), a2 = c_mul(c_sub(x0, x2), w1a);
    const float2 a1 = c_add(x1, x3), a3 = c_mul(c_sub(x1, x3), w1b);
    x[0] = c_add(a0, a1);
    x[ST] = c_mul(c_sub(a0, a1), w2);
    x[2 * ST] = c_add(a2, a3);
    x[3 * ST] = c_mul2(c_sub(a2, a3), w2);
  } else {
    const float2 t1 = c_mulc(x1, w2), t3 = c_mulc(x3, w2);
    const float2 a0 = c_add(x0, t1), a1 = c_sub(x0, t1);
    const float2 a2 = c_add(x2, t3), a3 = c_sub(x2, t3);
    const float2 t2 = c_mulc(a2, w1a), t4 = c_mulc(a3, w1b);
    x[0] = c_add(a0, t2);
    x[2 * ST] = c_sub(a0, t2);
    x[ST] = c_add(a1, t4);
    x[3 * ST] = c_sub(a1, t4);
  }
}

// The radix-2 stage of span 1 (twiddle 1).
__device__ __forceinline__ void last_stage(float2* x) {
  const float2 x0 = x[0], x1 = x[1];
  x[0] = c_add(x0, x1);
  x[1] = c_sub(x0, x1);
}

// G radix-2 stages (the lowest of them of span 2^(top - G)) on the 2^G elements of a
// thread, positions ... + i 2^(top - G) + j of a line of 2^lgn; tw[j] = exp(-2 pi i j / n)
template <int G, bool INV>
__device__ __forceinline__ void stages(float2 (&x)[1 << G], const float2* tw, int j, int lgn,
                                       int top) {
  constexpr int R = 1 << G;
  if constexpr (G == 1) {
    last_stage(x);
  } else {
    const int m = 1 << (top - 2), lgs = lgn - top;   // the upper pair: spans 2 m and m
    auto upper = [&] {
#pragma unroll
      for (int i = 0; i < R / 4; ++i) {
        const int jj = j + (i << (top - G));
        pair_stage<INV, R / 4>(x + i, tw[jj << lgs], tw[(jj + m) << lgs], tw[(2 * jj) << lgs]);
      }
    };
    auto lower = [&] {
      if constexpr (G == 4) {
        const int l2 = lgs + 2, m2 = m >> 2;
        const float2 w1a = tw[j << l2], w1b = tw[(j + m2) << l2], w2 = tw[(2 * j) << l2];
#pragma unroll
        for (int g = 0; g < 4; ++g) pair_stage<INV, 1>(x + 4 * g, w1a, w1b, w2);
      }
      if constexpr (G == 3) {
#pragma unroll
        for (int g = 0; g < 4; ++g) last_stage(x + 2 * g);
      }
    };
    if (INV) {
      lower();
      upper();
    } else {
      upper();
      lower();
    }
  }
}

// Stages of the group that starts at span 2^(top - 1): the pairs of stages from the top,
// a last single one (odd lg) in a group with the pair above it.
// The x lines end in a group of at most 8, since the curl holds it of all three components.
enum Axis { YZ, X };
template <Axis AX>
__host__ __device__ constexpr int group(int top) {
  return top >= 6 ? 4 : (top == 5 || (AX == X && top == 4) ? 2 : top);
}

// x[i] = ld(l, p0 + i 2^lgm); FP64 values are all loaded before the first conversion (its rare
// branch would keep the later loads behind it)
template <int R, class Ld>
__device__ __forceinline__ void load_all(float2 (&x)[R], Ld ld, int l, int p0, int lgm) {
  if constexpr (sizeof(ld(0, 0)) == sizeof(double2)) {
    double2 v[R];
#pragma unroll
    for (int i = 0; i < R; ++i) v[i] = ld(l, p0 + (i << lgm));
#pragma unroll
    for (int i = 0; i < R; ++i) x[i] = f64_to_f32(v[i]);
  } else {
#pragma unroll
    for (int i = 0; i < R; ++i) x[i] = ld(l, p0 + (i << lgm));
  }
}

// One group of stages of every line: item u -> (line l, position base p0, twiddle index j)
// by map, element i at position p0 + i 2^(top - G); ld and sv move them.
template <int G, bool INV, class Map, class Ld, class Sv>
__device__ __forceinline__ void group_pass(int items, int lgn, int top, const float2* tw, Map map,
                                           Ld ld, Sv sv) {
  const int lgm = top - G;
  for (int u = threadIdx.x; u < items; u += blockDim.x) {
    int l, r;
    map(u, G, l, r);
    const int j = r & ((1 << lgm) - 1), p0 = ((r >> lgm) << top) + j;
    float2 x[1 << G];
    load_all<1 << G>(x, ld, l, p0, lgm);
    stages<G, INV>(x, tw, j, lgn, top);
#pragma unroll
    for (int i = 0; i < (1 << G); ++i) sv(l, p0 + (i << lgm), x[i]);
  }
}

template <bool INV, Axis AX = YZ, class Map, class Ld, class Sv>
__device__ __forceinline__ void any_group(int points, int lgn, int top, const float2* tw, Map map,
                                          Ld ld, Sv sv) {
  switch (group<AX>(top)) {
    case 4: group_pass<4, INV>(points >> 4, lgn, top, tw, map, ld, sv); break;
    case 3: group_pass<3, INV>(points >> 3, lgn, top, tw, map, ld, sv); break;
    case 2: group_pass<2, INV>(points >> 2, lgn, top, tw, map, ld, sv); break;
    default: group_pass<1, INV>(points >> 1, lgn, top, tw, map, ld, sv); break;
  }
}

struct PlaneArgs {
  int lgy, lgz, ny, nz, nx;
  long long N, P;                 // grid points, points per (y, z) plane
  const float2* twy;              // exp(-2 pi i j / ny), j < ny (global)
  const float2* twz;
};

// padded plane of P elements in shared memory: one slot after each row of nz, so that
// rows start on successive banks
__host__ __device__ inline long long plane_slots(long long P, int lgz) { return P + (P >> lgz); }

// The plane in shared memory with its twiddles, and how items of its passes lie on threads.
struct Plane {
  float2 *a, *sty, *stz;
  int lgy, lgz, row;              // slots per row
  __device__ explicit Plane(const PlaneArgs& A, unsigned char* sm)
      : a(reinterpret_cast<float2*>(sm)), lgy(A.lgy), lgz(A.lgz), row(A.nz + 1) {
    sty = a + plane_slots(A.P, A.lgz);
    stz = sty + (A.ny >> 1);
    for (int j = threadIdx.x; j < (A.ny >> 1); j += blockDim.x) sty[j] = A.twy[j];
    for (int j = threadIdx.x; j < (A.nz >> 1); j += blockDim.x) stz[j] = A.twz[j];
  }
  // along y: consecutive threads on consecutive columns
  __device__ auto ymap() const {
    return [lgz = lgz](int u, int, int& l, int& r) {
      l = u & ((1 << lgz) - 1);
      r = u >> lgz;
    };
  }
  // along z within shared memory: consecutive threads on consecutive rows
  __device__ auto zmap() const {
    return [lgy = lgy](int u, int, int& l, int& r) {
      l = u & ((1 << lgy) - 1);
      r = u >> lgy;
    };
  }
  // along z with a global side: consecutive threads on the 2^(lgz - G) consecutive points
  // of a row, then (half a warp) on rows as far apart as that, for successive banks
  __device__ auto zmap_global() const {
    return [lgy = lgy, lgz = lgz](int u, int G, int& l, int& r) {
      const int lgj = lgz - G;
      r = u & ((1 << lgj) - 1);
      l = u >> lgj;
      if (lgj < 4 && lgy >= 4) {
        const int h = 4 - lgj, q = l & 15;
        l = (l & ~15) | ((q & ((1 << h) - 1)) << lgj) | (q >> h);
      }
    };
  }
  __device__ auto yat() const {
    return [a = a, row = row](int l, int p) -> float2& { return a[p * row + l]; };
  }
  __device__ auto zat() const {
    return [a = a, row = row](int l, int p) -> float2& { return a[l * row + p]; };
  }
  // forward: the groups of z after the first, then y; the last one to W
  __device__ void forward_rest(const PlaneArgs& A, float2* W) const {
    const auto z = zat();
    const auto y = yat();
    const int P = (int)A.P;
    for (int top = lgz - group<YZ>(lgz); top > 0; top -= group<YZ>(top)) {
      __syncthreads();
      any_group<false>(P, lgz, top, stz, zmap(), z, [&](int l, int p, float2 v) { z(l, p) = v; });
    }
    for (int top = lgy; top > 0; top -= group<YZ>(top)) {
      __syncthreads();
      if (top > group<YZ>(top))
        any_group<false>(P, lgy, top, sty, ymap(), y, [&](int l, int p, float2 v) { y(l, p) = v; });
      else
        any_group<false>(P, lgy, top, sty, ymap(), y,
                         [&](int l, int p, float2 v) { W[(p << lgz) + l] = v; });
    }
  }
};

// pass A: plane (x = blockIdx.x, component blockIdx.y) of the FP64 field F -> W
// (FP64 -> FP32 on the integer pipe: the FP64 pipe is ~1/64 of the FP32 rate here)
__global__ void __launch_bounds__(kPlaneThreads, 1) k_plane_fwd(PlaneArgs A, const double2* F,
                                                                float2* W) {
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smraw[];
  const Plane S(A, smraw);
  const long long base = blockIdx.y * A.N + blockIdx.x * A.P;
  F += base;
  __syncthreads();   // twiddles
  const auto z = S.zat();
  any_group<false>((int)A.P, A.lgz, A.lgz, S.stz, S.zmap_global(),
                   [&](int l, int p) { return F[(l << A.lgz) + p]; },
                   [&](int l, int p, float2 v) { z(l, p) = v; });
  S.forward_rest(A, W + base);
}

// The middle of pass B on the 2^G bottom positions of an x line of all three components:
// the last forward stages, the curl, the first inverse stages.  qb*: the wavenumbers of the
// bit-reversed positions as FP32 pairs (hi, lo): k f = fmaf(hi, f, lo f), one rounding per
// product (an FP32 wavenumber alone is up to 6e-8 off, a fixed phase-velocity error of its
// mode)
template <int G, class Ld, class Sv>
__device__ __forceinline__ void curl_group(const PlaneArgs& A, int lgx, int tl, long long b0,
                                           const float2* tw, const float2* qbx, const float2* qby,
                                           const float2* qbz, Ld ld, Sv sv) {
  constexpr int R = 1 << G;
  for (int u = threadIdx.x; u < (tl << lgx) >> G; u += blockDim.x) {
    const int c = u & (tl - 1), p0 = (u / tl) << G;   // tl is a power of two
    const long long col = b0 + c;
    const float2 ky = qby[(int)(col >> A.lgz)], kz = qbz[(int)(col & (A.nz - 1))];
    float2 x[3][R];
#pragma unroll
    for (int f = 0; f < 3; ++f) {
#pragma unroll
      for (int i = 0; i < R; ++i) x[f][i] = ld(f, c, p0 + i);
      stages<G, false>(x[f], tw, 0, lgx, G);
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const float2 kx = qbx[p0 + i];
      const float2 fx = x[0][i], fy = x[1][i], fz = x[2][i];
      auto km = [](float2 k, float f) { return fmaf(k.x, f, k.y * f); };
      // i (k x F)
      const float cxr = km(ky, fz.x) - km(kz, fy.x), cxi = km(ky, fz.y) - km(kz, fy.y);
      const float cyr = km(kz, fx.x) - km(kx, fz.x), cyi = km(kz, fx.y) - km(kx, fz.y);
      const float czr = km(kx, fy.x) - km(ky, fx.x), czi = km(kx, fy.y) - km(ky, fx.y);
      x[0][i] = make_float2(-cxi, cxr);
      x[1][i] = make_float2(-cyi, cyr);
      x[2][i] = make_float2(-czi, czr);
    }
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      stages<G, true>(x[f], tw, 0, lgx, G);
#pragma unroll
      for (int i = 0; i < R; ++i) sv(f, c, p0 + i, x[f][i]);
    }
  }
}

// pass B: the x lines of tl consecutive (y, z) columns of all three components;
// shared memory [x][component][column]
__global__ void __launch_bounds__(kXThreads, 2) k_x_curl_ip(PlaneArgs A, float2* W, int lgx, int tl,
                                                            const float2* twx, const float2* qbx,
                                                            const float2* qby, const float2* qbz) {
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smraw[];
  const int nx = 1 << lgx, w3 = 3 * tl;
  float2* a = reinterpret_cast<float2*>(smraw);
  float2* stx = a + (size_t)nx * w3;
  for (int j = threadIdx.x; j < (nx >> 1); j += blockDim.x) stx[j] = twx[j];
  const long long b0 = (long long)blockIdx.x * tl;
  W += b0;
  const auto wat = [&](int f, int c, int p) -> float2& { return W[f * A.N + p * A.P + c]; };
  const auto sat = [&](int f, int c, int p) -> float2& { return a[p * w3 + f * tl + c]; };
  // lines of one component: consecutive threads on consecutive columns
  const auto map = [&](int u, int, int& l, int& r) {
    l = u & (tl - 1);
    r = u / tl;
  };
  __syncthreads();   // twiddles
  int top = lgx;
  for (; top > group<X>(top); top -= group<X>(top)) {
    for (int f = 0; f < 3; ++f)
      if (top == lgx)
        any_group<false, X>(tl << lgx, lgx, top, stx, map, [&](int l, int p) { return wat(f, l, p); },
                         [&](int l, int p, float2 v) { sat(f, l, p) = v; });
      else
        any_group<false, X>(tl << lgx, lgx, top, stx, map, [&](int l, int p) { return sat(f, l, p); },
                         [&](int l, int p, float2 v) { sat(f, l, p) = v; });
    __syncthreads();
  }
  const auto ws = [&](int f, int c, int p, float2 v) { wat(f, c, p) = v; };
  const auto ss = [&](int f, int c, int p, float2 v) { sat(f, c, p) = v; };
  if (top == lgx) {   // at most 8 points: nothing goes through shared memory
    switch (top) {
      case 3: curl_group<3>(A, lgx, tl, b0, stx, qbx, qby, qbz, wat, ws); break;
      case 2: curl_group<2>(A, lgx, tl, b0, stx, qbx, qby, qbz, wat, ws); break;
      default: curl_group<1>(A, lgx, tl, b0, stx, qbx, qby, qbz, wat, ws); break;
    }
    return;
  }
  switch (top) {   // 2 or 3 below a group of its own
    case 3: curl_group<3>(A, lgx, tl, b0, stx, qbx, qby, qbz, sat, ss); break;
    default: curl_group<2>(A, lgx, tl, b0, stx, qbx, qby, qbz, sat, ss); break;
  }
  // the inverse groups above, in the order of the forward ones turned round
  while (top < lgx) {
    int up = lgx;
    while (up - group<X>(up) > top) up -= group<X>(up);
    __syncthreads();
    for (int f = 0; f < 3; ++f)
      if (up == lgx)
        any_group<true, X>(tl << lgx, lgx, up, stx, map, [&](int l, int p) { return sat(f, l, p); },
                        [&](int l, int p, float2 v) { wat(f, l, p) = v; });
      else
        any_group<true, X>(tl << lgx, lgx, up, stx, map, [&](int l, int p) { return sat(f, l, p); },
                        [&](int l, int p, float2 v) { sat(f, l, p) = v; });
    top = up;
  }
}

// The end of pass C on one thread's 2^G points of a z line: the last inverse stages, then
// out (+)= ...: the update of Upd (the masks per axis); with fwd_next the updated values
// continue as the first stages of the next curl.  The increment a v / N - ja J is formed in
// FP32 (v is the FP32 transform; a / N and ja as FP32 pairs, J rounded to FP32 on the integer
// pipe) and added to the FP64 field: one FP64 add per component; the mask multiplies only
// where it is not 1.
template <int G>
__device__ __forceinline__ void update_group(const PlaneArgs& A, const Plane& S, const Upd& U,
                                             long long base, int x, int fwd_next) {
  constexpr int R = 1 << G;
  const auto z = S.zat();
  const auto map = S.zmap_global();
  const double mx = U.m0 ? U.m0[x] : 1.0;
  const bool xin = min(x, A.nx - 1 - x) >= U.nabc[0];
  const int lgm = A.lgz - G;
  double2* out = U.out + base;
  const double2* J = U.J ? U.J + base : nullptr;
  for (int u = threadIdx.x; u < (int)A.P >> G; u += blockDim.x) {
    int y, j;
    map(u, G, y, j);
    float2 v[R];
#pragma unroll
    for (int i = 0; i < R; ++i) v[i] = z(y, j + (i << lgm));
    stages<G, true>(v, S.stz, j, A.lgz, A.lgz);
    const bool yin = xin && min(y, A.ny - 1 - y) >= U.nabc[1];
    constexpr int B = R < 4 ? R : 4;   // FP64 loads of B points before their updates
#pragma unroll
    for (int i0 = 0; i0 < R; i0 += B) {
      double2 o[B], jv[B];
#pragma unroll
      for (int q = 0; q < B; ++q) {
        const int i = (y << A.lgz) + j + ((i0 + q) << lgm);
        o[q] = U.store ? make_double2(0.0, 0.0) : out[i];
        jv[q] = J ? J[i] : make_double2(0.0, 0.0);
      }
#pragma unroll
      for (int q = 0; q < B; ++q) {
        const int zi = j + ((i0 + q) << lgm);
        const float2 w = v[i0 + q];
        float ix = fmaf(w.x, U.af[0], w.x * U.af[1]), iy = fmaf(w.y, U.af[0], w.y * U.af[1]);
        if (J) {
          const float2 jf = f64_to_f32(jv[q]);
          ix -= fmaf(jf.x, U.jf[0], jf.x * U.jf[1]);
          iy -= fmaf(jf.y, U.jf[0], jf.y * U.jf[1]);
        }
        double2 r = make_double2(o[q].x + f32_to_f64(ix), o[q].y + f32_to_f64(iy));
        // FP64 only inside the absorbing layers (integer test of the position)
        if (U.m0 && (!yin || min(zi, A.nz - 1 - zi) < U.nabc[2])) {
          const double m = mx * U.m1[y] * U.m2[zi];
          r.x *= m;
          r.y *= m;
        }
        out[(y << A.lgz) + zi] = r;
        v[i0 + q] = f64_to_f32(r);
      }
    }
    if (fwd_next) {
      stages<G, false>(v, S.stz, j, A.lgz, A.lgz);
#pragma unroll
      for (int i = 0; i < R; ++i) z(y, j + (i << lgm)) = v[i];
    }
  }
}

// pass C: inverse along y and z of plane (x, component), the update, and with fwd_next pass A
// of the next curl (W overwritten with its transform: the block owns its plane of W)
__global__ void __launch_bounds__(kPlaneThreads, 1) k_plane_inv(PlaneArgs A, float2* W, Upd U,
                                                                int fwd_next) {
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smraw[];
  const Plane S(A, smraw);
  const int x = blockIdx.x, P = (int)A.P;
  const long long base = blockIdx.y * A.N + x * A.P;
  float2* w = W + base;
  const auto z = S.zat();
  const auto y = S.yat();
  // y from the lowest group up, the first one from W
  for (int top = 0; top < A.lgy;) {
    int up = A.lgy;
    while (up - group<YZ>(up) > top) up -= group<YZ>(up);
    __syncthreads();
    if (top == 0)
      any_group<true>(P, A.lgy, up, S.sty, S.ymap(),
                      [&](int l, int p) { return w[(p << A.lgz) + l]; },
                      [&](int l, int p, float2 v) { y(l, p) = v; });
    else
      any_group<true>(P, A.lgy, up, S.sty, S.ymap(), y,
                      [&](int l, int p, float2 v) { y(l, p) = v; });
    top = up;
  }
  for (int top = 0; top < A.lgz - group<YZ>(A.lgz);) {
    int up = A.lgz;
    while (up - group<YZ>(up) > top) up -= group<YZ>(up);
    __syncthreads();
    any_group<true>(P, A.lgz, up, S.stz, S.zmap(), z, [&](int l, int p, float2 v) { z(l, p) = v; });
    top = up;
  }
  __syncthreads();
  switch (group<YZ>(A.lgz)) {
    case 4: update_group<4>(A, S, U, base, x, fwd_next); break;
    case 3: update_group<3>(A, S, U, base, x, fwd_next); break;
    case 2: update_group<2>(A, S, U, base, x, fwd_next); break;
    default: update_group<1>(A, S, U, base, x, fwd_next); break;
  }
  if (fwd_next) S.forward_rest(A, w);   // block-uniform
}

bool pow2(int v) { return v >= 2 && v <= 1024 && (v & (v - 1)) == 0; }

// tl lines per block within the shared-memory budget (two ping-pong buffers of nf
// fields x n x tl elements), tl <= 8 and dividing inner
int lines_per_block(int n, int nf, size_t elem, int inner) {
  int tl = 8;
  while (tl > 1 && (2 * (size_t)nf * n * tl * elem > (size_t)kSmemMax || inner % tl)) tl >>= 1;
  return tl;
}

template <typename T>
int run_line_pass(SbePstd3* p, int axis, int dir, int nf, const double2* in64, T* W,
                  const Upd& U, cudaStream_t s) {
  Pass P{};
  P.n = p->n[axis];
  P.lg = ilog2i(P.n);
  P.s = axis == 2 ? 1 : (axis == 1 ? p->n[2] : p->n[1] * p->n[2]);
  P.inner = P.s;
  P.N = p->N;
  P.nf = nf;
  P.dir = dir;
  P.tw = p->tw[axis];
  P.twf = p->twf[axis];
  const int lines = (int)(p->N / P.n);
  P.tl = P.s == 1 ? 8 : lines_per_block(P.n, 1, sizeof(T), P.inner);
  if (P.s == 1)
    while (P.tl > 1 && 2 * (size_t)P.n * P.tl * sizeof(T) > (size_t)kSmemMax) P.tl >>= 1;
  P.lgtl = ilog2i(P.tl);
  const size_t smem = 2 * (size_t)P.n * P.tl * sizeof(T);
  const dim3 grid(lines / P.tl, nf);
  launch(k_line_pass<T>, grid, kThreads, smem, s, P, in64, W, U);
  return cuda_check(cudaGetLastError(), "pstd3 line pass");
}

template <typename T>
int run_x_curl(SbePstd3* p, T* W, cudaStream_t s) {
  Pass P{};
  P.n = p->n[0];
  P.lg = ilog2i(P.n);
  P.s = p->n[1] * p->n[2];
  P.inner = P.s;
  P.N = p->N;
  P.tw = p->tw[0];
  P.twf = p->twf[0];
  P.tl = lines_per_block(P.n, 3, sizeof(T), P.inner);
  P.lgtl = ilog2i(P.tl);
  const size_t smem = 2 * 3 * (size_t)P.n * P.tl * sizeof(T);
  launch(k_x_curl<T>, P.s / P.tl, kThreads, smem, s, P, W, p->q[1], p->q[2], p->q[0], p->n[2]);
  return cuda_check(cudaGetLastError(), "pstd3 curl pass");
}

Upd upd_store(SbePstd3* p) {
  Upd U{};
  U.nx = p->n[0];
  U.ny = p->n[1];
  U.nz = p->n[2];
  return U;
}

// out (+)= curl F: a, ja, J, masked as in Upd (store = 1: out = curl F).
template <typename T>
int curl_pipeline(SbePstd3* p, const double2* F, double2* out, double a, const double2* J,
                  double ja, bool masked, int store, cudaStream_t s) {
  T* W = static_cast<T*>(p->work);
  Upd none = upd_store(p);
  int rc = run_line_pass<T>(p, 2, -1, 3, F, W, none, s);
  if (!rc) rc = run_line_pass<T>(p, 1, -1, 3, nullptr, W, none, s);
  if (!rc) rc = run_x_curl<T>(p, W, s);
  if (!rc) rc = run_line_pass<T>(p, 1, +1, 3, nullptr, W, none, s);
  if (rc) return rc;
  Upd U = upd_store(p);
  U.out = out;
  U.a = a;
  U.J = J;
  U.ja = ja;
  U.store = store;
  if (masked) {
    U.m0 = p->mask[0];
    U.m1 = p->mask[1];
    U.m2 = p->mask[2];
  }
  return run_line_pass<T>(p, 2, +1, 3, nullptr, W, U, s);
}

int curl_any(SbePstd3* p, const double2* F, double2* out, double a, const double2* J, double ja,
             bool masked, int store, cudaStream_t s) {
  return p->fp32 ? curl_pipeline<float2>(p, F, out, a, J, ja, masked, store, s)
                 : curl_pipeline<double2>(p, F, out, a, J, ja, masked, store, s);
}

bool is_masked(const SbePstd3* p) { return p->n_abc[0] > 0 || p->n_abc[1] > 0 || p->n_abc[2] > 0; }

// ---- the three-pass curl (FP32 work, planes in shared memory) -----------------
bool planes_fit(const SbePstd3* p) { return p->fp32 && (long long)p->n[1] * p->n[2] <= kPlaneMax; }

PlaneArgs plane_args(const SbePstd3* p) {
  PlaneArgs A{};
  A.nx = p->n[0];
  A.ny = p->n[1];
  A.nz = p->n[2];
  A.lgy = ilog2i(A.ny);
  A.lgz = ilog2i(A.nz);
  A.N = p->N;
  A.P = (long long)A.ny * A.nz;
  A.twy = p->twf[1];
  A.twz = p->twf[2];
  return A;
}

size_t plane_smem(const PlaneArgs& A) {
  return sizeof(float2) * ((size_t)plane_slots(A.P, A.lgz) + (A.ny >> 1) + (A.nz >> 1));
}

// 16 points per thread, so that small planes share an SM
int plane_threads(const PlaneArgs& A) {
  return (int)std::min<long long>(kPlaneThreads, std::max<long long>(32, A.P / 16));
}

// x-pass columns per block: the three components' x lines of tl columns within
// kXSmem, tl <= 16 and dividing the plane
int x_lines(const SbePstd3* p) {
  const long long P = (long long)p->n[1] * p->n[2];
  int tl = 16;
  while (tl > 1 && ((size_t)3 * p->n[0] * tl * sizeof(float2) > (size_t)kXSmem || P % tl)) tl >>= 1;
  return tl;
}

int plane_pass_a(SbePstd3* p, const double2* F, cudaStream_t s) {
  const PlaneArgs A = plane_args(p);
  launch(k_plane_fwd, dim3(A.nx, 3), plane_threads(A), plane_smem(A), s, A, F,
         static_cast<float2*>(p->work));
  return cuda_check(cudaGetLastError(), "pstd3 plane pass");
}

int plane_pass_b(SbePstd3* p, cudaStream_t s) {
  const PlaneArgs A = plane_args(p);
  const int tl = x_lines(p), nx = p->n[0];
  const size_t smem = sizeof(float2) * ((size_t)3 * nx * tl + (nx >> 1));
  launch(k_x_curl_ip, (unsigned)(A.P / tl), kXThreads, smem, s, A, static_cast<float2*>(p->work),
         ilog2i(nx), tl, p->twf[0], p->qb[0], p->qb[1], p->qb[2]);
  return cuda_check(cudaGetLastError(), "pstd3 x pass");
}

int plane_pass_c(SbePstd3* p, const Upd& U, int fwd_next, cudaStream_t s) {
  const PlaneArgs A = plane_args(p);
  launch(k_plane_inv, dim3(A.nx, 3), plane_threads(A), plane_smem(A), s, A,
         static_cast<float2*>(p->work), U, fwd_next);
  return cuda_check(cudaGetLastError(), "pstd3 plane pass");
}

Upd upd_for(SbePstd3* p, double2* out, double a, const double2* J, double ja, bool masked,
            int store) {
  Upd U = upd_store(p);
  U.out = out;
  U.a = a;
  U.J = J;
  U.ja = ja;
  U.store = store;
  if (masked) {
    U.m0 = p->mask[0];
    U.m1 = p->mask[1];
    U.m2 = p->mask[2];
  }
  for (int ax = 0; ax < 3; ++ax) U.nabc[ax] = p->n_abc[ax];
  // FP32 pairs of the plane path: the curl arrives as N curl (N a power of two)
  const double an = (store ? 1.0 : a) / (double)p->N;
  U.af[0] = (float)an;
  U.af[1] = (float)(an - (double)U.af[0]);
  U.jf[0] = (float)ja;
  U.jf[1] = (float)(ja - (double)U.jf[0]);
  return U;
}

// out (+)= a curl F ...: the three-pass form when the planes fit, else five passes
int curl_best(SbePstd3* p, const double2* F, double2* out, double a, const double2* J, double ja,
              bool masked, int store, cudaStream_t s) {
  if (!planes_fit(p)) return curl_any(p, F, out, a, J, ja, masked, store, s);
  int rc = plane_pass_a(p, F, s);
  if (!rc) rc = plane_pass_b(p, s);
  if (!rc) rc = plane_pass_c(p, upd_for(p, out, a, J, ja, masked, store), 0, s);
  return rc;
}

}  // namespace

// The H half-step of a field step, leaving the work array ready for the E half-step
// of the same step: with planes in shared memory the H update's last pass continues
// with the first pass of curl H on the new H.
int pstd3_update_h_fwd(SbePstd3* p, const double2* E, double2* H, double dt, cudaStream_t s) {
  if (!planes_fit(p))
    return curl_any(p, E, H, -dt / kMu0, nullptr, 0.0, is_masked(p), 0, s);
  int rc = plane_pass_a(p, E, s);
  if (!rc) rc = plane_pass_b(p, s);
  if (!rc) rc = plane_pass_c(p, upd_for(p, H, -dt / kMu0, nullptr, 0.0, is_masked(p), 0), 1, s);
  return rc;
}

// The E half-step after pstd3_update_h_fwd on the same H, with nothing else using the
// work array in between.
int pstd3_update_e_from_work(SbePstd3* p, double2* E, const double2* H, const double2* J,
                             double dt, cudaStream_t s) {
  const double ie = dt / (kEps0 * p->epsr);
  if (!planes_fit(p)) return curl_any(p, H, E, ie, J, ie, is_masked(p), 0, s);
  int rc = plane_pass_b(p, s);
  if (!rc) rc = plane_pass_c(p, upd_for(p, E, ie, J, ie, is_masked(p), 0), 0, s);
  return rc;
}

}  // namespace sbe

using namespace sbe;

extern "C" {

int sbe_pstd3_create(const SbePstd3Desc* d, void* stream, SbePstd3** out) {
  if (!d || !out) return fail(SBE_ERR_ARG, "sbe_pstd3_create: null");
  *out = nullptr;
  for (int a = 0; a < 3; ++a) {
    if (!pow2(d->n[a]))
      return fail(SBE_ERR_UNSUPPORTED, "sbe_pstd3_create: every axis must be a power of two in "
                                       "[2, 1024]");
    if (!(d->d[a] > 0) || d->n_abc[a] < 0 || 2 * d->n_abc[a] > d->n[a])
      return fail(SBE_ERR_ARG, "sbe_pstd3_create: bad spacing or absorbing width");
  }
  if (!(d->epsr > 0) || d->abc_strength < 0) return fail(SBE_ERR_ARG, "sbe_pstd3_create: bad epsr");
  SbePstd3* p = new SbePstd3();
  for (int a = 0; a < 3; ++a) {
    p->n[a] = d->n[a];
    p->n_abc[a] = d->n_abc[a];
    p->d[a] = d->d[a];
  }
  p->fp32 = d->fp32_work ? 1 : 0;
  p->epsr = d->epsr;
  p->abc = d->abc_strength;
  p->N = (long long)p->n[0] * p->n[1] * p->n[2];
  size_t tab = 0;
  for (int a = 0; a < 3; ++a)
    tab += ((3 * sizeof(double) + sizeof(double2) + 2 * sizeof(float2)) * p->n[a] + 1536);
  // work: ten FP64 complex fields (the longitudinal-field spectra; the curl uses three)
  const size_t work = sizeof(double2) * 10 * (size_t)p->N;
  if (cudaMalloc(&p->arena, tab + work) != cudaSuccess) {
    delete p;
    return fail(SBE_ERR_OOM, "sbe_pstd3_create: device allocation");
  }
  char* b = static_cast<char*>(p->arena);
  auto take = [&](size_t bytes) {
    char* r = b;
    b += (bytes + 255) / 256 * 256;
    return r;
  };
  cudaStream_t s = as_stream(stream);
  for (int a = 0; a < 3; ++a) {
    const int n = p->n[a];
    p->x[a] = reinterpret_cast<double*>(take(sizeof(double) * n));
    p->q[a] = reinterpret_cast<double*>(take(sizeof(double) * n));
    p->mask[a] = reinterpret_cast<double*>(take(sizeof(double) * n));
    p->tw[a] = reinterpret_cast<double2*>(take(sizeof(double2) * n));
    p->twf[a] = reinterpret_cast<float2*>(take(sizeof(float2) * n));
    p->qb[a] = reinterpret_cast<float2*>(take(sizeof(float2) * n));
    k_tables3<<<(n + 127) / 128, 128, 0, s>>>(n, p->d[a], p->x[a], p->q[a], p->tw[a], p->twf[a],
                                             p->qb[a], p->mask[a], p->n_abc[a], p->abc);
  }
  p->work = take(work);
  int rc = cuda_check(cudaGetLastError(), "sbe_pstd3_create");
  if (!rc) {
    const int smem = kSmemMax + 1024;
    cudaFuncSetAttribute(k_line_pass<double2>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    cudaFuncSetAttribute(k_line_pass<float2>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    cudaFuncSetAttribute(k_x_curl<double2>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    cudaFuncSetAttribute(k_plane_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    cudaFuncSetAttribute(k_plane_inv, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    cudaFuncSetAttribute(k_x_curl_ip, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    rc = cuda_check(cudaFuncSetAttribute(k_x_curl<float2>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
                    "sbe_pstd3_create: shared memory");
  }
  if (!rc) rc = cuda_check(cudaStreamSynchronize(s), "sbe_pstd3_create: tables");
  if (rc) {
    cudaFree(p->arena);
    delete p;
    return rc;
  }
  *out = p;
  return SBE_OK;
}

int sbe_pstd3_destroy(SbePstd3* p) {
  if (!p) return SBE_OK;
  cudaFree(p->arena);
  delete p;
  return SBE_OK;
}

int sbe_pstd3_grid(SbePstd3* p, int axis, double* x, double* q, void* stream) {
  if (!p || axis < 0 || axis > 2) return fail(SBE_ERR_ARG, "sbe_pstd3_grid: bad arguments");
  cudaStream_t s = as_stream(stream);
  const size_t b = sizeof(double) * p->n[axis];
  if (x) cudaMemcpyAsync(x, p->x[axis], b, cudaMemcpyDeviceToDevice, s);
  if (q) cudaMemcpyAsync(q, p->q[axis], b, cudaMemcpyDeviceToDevice, s);
  return cuda_check(cudaGetLastError(), "sbe_pstd3_grid");
}

int sbe_pstd3_curl(SbePstd3* p, const double* F, double* out, void* stream) {
  if (!p || !F || !out) return fail(SBE_ERR_ARG, "sbe_pstd3_curl: null");
  return curl_best(p, (const double2*)F, (double2*)out, 1.0, nullptr, 0.0, false, 1,
                   as_stream(stream));
}

int sbe_pstd3_update_h(SbePstd3* p, const double* E, double* H, double dt, void* stream) {
  if (!p || !E || !H) return fail(SBE_ERR_ARG, "sbe_pstd3_update_h: null");
  return curl_best(p, (const double2*)E, (double2*)H, -dt / kMu0, nullptr, 0.0, is_masked(p), 0,
                   as_stream(stream));
}

int sbe_pstd3_update_e(SbePstd3* p, double* E, const double* H, const double* J, double dt,
                       void* stream) {
  if (!p || !E || !H) return fail(SBE_ERR_ARG, "sbe_pstd3_update_e: null");
  const double ie = dt / (kEps0 * p->epsr);
  return curl_best(p, (const double2*)H, (double2*)E, ie, (const double2*)J, ie, is_masked(p), 0,
                   as_stream(stream));
}

int sbe_pstd3_step(SbePstd3* p, double* E, double* H, const double* J, double dt, void* stream) {
  if (!p) return fail(SBE_ERR_ARG, "sbe_pstd3_step: null");
  // stability of the spectral leapfrog: v dt |q|max / 2 <= 1
  const double v = 299792458.0 / std::sqrt(p->epsr);
  double qm = 0.0;
  for (int a = 0; a < 3; ++a) qm += (kPi / p->d[a]) * (kPi / p->d[a]);
  if (v * dt * std::sqrt(qm) / 2.0 > 1.0)
    return fail(SBE_ERR_ARG, "sbe_pstd3_step: dt above the stability limit 2 / (v |q|max)");
  if (!E || !H) return fail(SBE_ERR_ARG, "sbe_pstd3_step: null");
  cudaStream_t s = as_stream(stream);
  int rc = pstd3_update_h_fwd(p, (const double2*)E, (double2*)H, dt, s);
  if (rc) return rc;
  return pstd3_update_e_from_work(p, (double2*)E, (const double2*)H, (const double2*)J, dt, s);
}

// rhoPJ.py:703-880 ElongfromRho with the caller's wavenumber tables (the reference
// passes its centred GetKxArray/GetKyArray/GetKzArray, typespace.py:958-1030): FP64
// forward transforms of rho, Px, Py, Pz (P_k receives the transformed P, as the
// reference leaves it in its inputs; may be NULL), the k-space terms and ten FP64
// inverse transforms into out10 = [E_PRho x, y, z, E_P x, y, z, E_Rho x, y, z, rho_B].
int sbe_pstd3_elong(SbePstd3* p, const double* rho, const double* P3, const double* qx,
                    const double* qy, const double* qz, double* out10, double* P_k,
                    void* stream) {
  if (!p || !rho || !P3 || !qx || !qy || !qz || !out10)
    return fail(SBE_ERR_ARG, "sbe_pstd3_elong: null");
  cudaStream_t s = as_stream(stream);
  const long long N = p->N;
  double2* O = reinterpret_cast<double2*>(out10);
  // the four transforms in out10's first four fields (FP64 work: the reference's FFT)
  cudaMemcpyAsync(O, rho, sizeof(double2) * N, cudaMemcpyDeviceToDevice, s);
  cudaMemcpyAsync(O + N, P3, sizeof(double2) * 3 * N, cudaMemcpyDeviceToDevice, s);
  Upd none = upd_store(p);
  int rc = SBE_OK;
  for (int a = 2; a >= 0 && !rc; --a) rc = run_line_pass<double2>(p, a, -1, 4, nullptr, O, none, s);
  if (rc) return rc;
  if (P_k) cudaMemcpyAsync(P_k, O + N, sizeof(double2) * 3 * N, cudaMemcpyDeviceToDevice, s);
  double2* S = static_cast<double2*>(p->work);
  cudaMemcpyAsync(S, O, sizeof(double2) * 4 * N, cudaMemcpyDeviceToDevice, s);
  double q01[2];
  rc = cuda_check(cudaMemcpyAsync(q01, qx, sizeof(double) * 2, cudaMemcpyDeviceToHost, s),
                  "sbe_pstd3_elong: q");
  if (!rc) rc = cuda_check(cudaStreamSynchronize(s), "sbe_pstd3_elong: q");
  if (rc) return rc;
  const double small = (q01[1] - q01[0]) / 1e4;
  k_elong3<<<(unsigned)((N + 255) / 256), 256, 0, s>>>(N, p->n[1], p->n[2], S, O, qx, qy, qz,
                                                       small, 1.0 / (kEps0 * p->epsr));
  // inverse transforms of the ten spectra; the last pass divides by N
  for (int a = 0; a < 2 && !rc; ++a) rc = run_line_pass<double2>(p, a, +1, 10, nullptr, O, none, s);
  if (rc) return rc;
  Upd U = upd_store(p);
  U.out = O;
  U.store = 1;
  // the last pass reads the work array: move the spectra there first
  cudaMemcpyAsync(S, O, sizeof(double2) * 10 * N, cudaMemcpyDeviceToDevice, s);
  rc = run_line_pass<double2>(p, 2, +1, 10, nullptr, S, U, s);
  return rc ? rc : cuda_check(cudaGetLastError(), "sbe_pstd3_elong");
}

}  // extern "C"
