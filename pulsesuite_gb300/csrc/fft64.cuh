// FP64 Stockham transforms over shared memory.
#pragma once
#include "sbe_internal.cuh"

namespace sbe {

// 2^lgtr transforms of length 2^lg (2 points take the opening stage alone): element p of transform c at a[p ps + c cs];
// consecutive threads walk c (c_fast) or p.  dir -1: exp(-i ...), +1: exp(+i ...);
// tw[j] = exp(-2 pi i j / 2^lg).  Returns the buffer, a or b, that holds the result in natural
// order.  Radix 4 (an odd log length opens with a radix-2 stage): the two-wide FP64 pipe bounds
// transforms that fill the SMs, and against radix 2 four values take 28 operations instead of 32
// and half the sweeps, the first stage 16; fewer products also round less.  3-D step of
// 256 x 128 x 128 10.6 -> 8.65 ms, 128 x 64 x 64 1.23 -> 0.96, curl error 3.7e-16 -> 3.5e-16.  The
// single lines of the 1-D transforms stay in radix 2: with a warp to a line the instructions of
// a radix-4 stage follow one another at 64 clocks each (rows of 128 9.9 -> 14.3 us).
__device__ inline double2* fft64(double2* a, double2* b, int lg, int lgtr, int ps, int cs,
                                 bool c_fast, int dir, const double2* tw) {
  const int L = 1 << lg;
  const auto place = [&](int idx, int lgj, int& j, int& c) {
    if (c_fast) {
      c = idx & ((1 << lgtr) - 1);
      j = idx >> lgtr;
    } else {
      j = idx & ((1 << lgj) - 1);
      c = idx >> lgj;
    }
  };
  // (u + w v, u - w v), both signs straight from the products
  const auto pair = [](double2 u, double2 v, double2 w, double2& p, double2& m) {
    p.x = fma(v.x, w.x, fma(-v.y, w.y, u.x));
    p.y = fma(v.x, w.y, fma(v.y, w.x, u.y));
    m.x = fma(-v.x, w.x, fma(v.y, w.y, u.x));
    m.y = fma(-v.x, w.y, fma(-v.y, w.x, u.y));
  };
  int ns = 1;
  if (lg & 1) {
    const int half = L >> 1;
    for (int idx = threadIdx.x; idx < half << lgtr; idx += blockDim.x) {
      int j, c;
      place(idx, lg - 1, j, c);
      const double2 u = a[j * ps + c * cs], v = a[(j + half) * ps + c * cs];
      b[2 * j * ps + c * cs] = cadd(u, v);
      b[(2 * j + 1) * ps + c * cs] = csub(u, v);
    }
    __syncthreads();
    double2* t = a;
    a = b;
    b = t;
    ns = 2;
  }
  const int q4 = L >> 2;
  for (; ns < L; ns <<= 2) {
    const int tws = q4 / ns;
    for (int idx = threadIdx.x; idx < q4 << lgtr; idx += blockDim.x) {
      int j, c;
      place(idx, lg - 2, j, c);
      const int k = j & (ns - 1), o = ((j - k) << 2) + k;
      const double2* in = a + j * ps + c * cs;
      const double2 x0 = in[0], x1 = in[q4 * ps], x2 = in[2 * q4 * ps], x3 = in[3 * q4 * ps];
      double2 a0, a2, b0, b2;
      if (ns == 1) {
        a0 = cadd(x0, x2);
        a2 = csub(x0, x2);
        b0 = cadd(x1, x3);
        b2 = csub(x1, x3);
      } else {
        double2 w1 = tw[k * tws], w2 = tw[2 * k * tws], w3 = tw[3 * k * tws];
        if (dir > 0) {
          w1.y = -w1.y;
          w2.y = -w2.y;
          w3.y = -w3.y;
        }
        pair(x0, x2, w2, a0, a2);
        pair(cmul(x1, w1), x3, w3, b0, b2);
      }
      if (dir > 0) b2 = make_double2(-b2.x, -b2.y);
      double2* out = b + o * ps + c * cs;
      out[0] = cadd(a0, b0);
      out[ns * ps] = make_double2(a2.x + b2.y, a2.y - b2.x);
      out[2 * ns * ps] = csub(a0, b0);
      out[3 * ns * ps] = make_double2(a2.x - b2.y, a2.y + b2.x);
    }
    __syncthreads();
    double2* t = a;
    a = b;
    b = t;
  }
  return a;
}

}  // namespace sbe
