// FP64 matrix products on the tensor cores by exact integer slices (the splitting of
// Ozaki, Ogita, Oishi and Rump, "Error-free transformations of matrix multiplication",
// Numer. Algorithms 59, 2012), for the FP64 path's contractions.
//
// Every row of an operand (both operands K-major: rows of A and of B^T) is scaled by a
// power of two to integers v of 2-norm below 2^62 and cut into digits,
// v = sum_i d_i 2^(8 (7 - i)), i = 0..7, |d_i| <= 128 (|d_0| <= 65), which FP16 holds
// exactly.  A product of two digit planes over K <= 128 is an integer of magnitude at most
// 2^24, so the tensor core's FP32 accumulation is exact whatever its order; the planes with
// i + j = t share one accumulator (2 x 65 x 128 + 6 x 128^2 times 128 stays below 2^24).
// The planes with i + j > 7 are left out: they add about 2^-57 of the rows' norms at K =
// 1024.  By Cauchy-Schwarz the whole sum over K stays below 2^124, so the epilogue adds the
// accumulators modulo 2^64 in units of 2^62 and rounds once to FP64.
// The error of an element is therefore measured by the norms of the two rows that meet in it, not
// by its own terms: an operand whose rows hold a few large elements beside small ones that matter
// gives those to the caller's FP64 (f64_path.cu: the diagonals of C, D, Hee, Hhh).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <cstdint>

#include "fp_bits.cuh"

namespace sbe {
namespace f64s {

constexpr int NS = 8;           // digit planes of one real matrix
constexpr int BM = 128, BN = 64, BK = 32;
constexpr int CHUNK = 4;        // K blocks per accumulation (K = 128)
constexpr int kBadExp = 1 << 28;   // row with an infinity or a NaN: its products are NaN
constexpr int MAX_JOBS = 16;

// One real-component plane set: form slab layout [plane][batch][K block][row][32 halves],
// 64-byte rows swizzled as the tensor core's 64-byte K-major mode reads them.
__host__ __device__ inline int pad_rows(int r) { return (r + 127) / 128 * 128; }
__host__ __device__ inline int k_blocks(int k) { return (k + BK - 1) / BK; }
__host__ __device__ inline long long slab(int rows, int k) {
  return (long long)pad_rows(rows) * k_blocks(k) * BK;
}

// One product out = +-A op B: A (M rows) and B^T (N rows) as digit planes.  cplx: 16
// planes (re, im) each and separate re / im outputs; else 8 planes each.
struct Job {
  const __half *A, *B;              // plane 0 of the operand, batch entry 0
  long long a_plane, a_batch, b_plane, b_batch;   // strides (halves)
  int a_pad, b_pad;                 // padded rows
  const int *ea, *eb;               // row exponents, batch stride M resp. N
  int M, N, nkb, batch;
  int cplx, conj_a, conj_b, neg;
  int parts;                        // cuts of the K sequence, each its own output
  int band;                         // exchange: Nk of the shear (0: off)
  double* out;                      // + part * o_part + comp * o_comp + b * o_batch
  long long o_part, o_comp, o_batch;
  int ldo;
};

struct Launch {
  Job job[MAX_JOBS];
  int base[MAX_JOBS + 1];
  int njobs;
  int stall;                        // self-test: no operand arrives, every wait runs out
  int* err;                         // raised by a wait that gave up
};

// One operand form of the slicing pass: row r, column k is src[r ld + k], or src[k ld + r]
// when transposed, of a batch of complex matrices; add (real parts of a complex matrix, or
// null, not transposed) times add_f joins the imaginary part; with peel the elements r = k count
// as zero.
struct Form {
  const double2* src;
  const double2* add;
  int transpose, peel;
  __half* dst;      // plane 0, batch entry 0
  int* e;           // row exponents (batch stride rows)
};
struct SliceArgs {
  Form f[14];
  int rows, kdim, ld, batch;
  long long src_batch;          // elements between the matrices of a batch
  long long plane, dst_batch;   // halves
  double add_f;
};

#ifdef __CUDACC__
// x 2^(62 - E) rounded to an integer (|x| < 2^E)
__device__ __forceinline__ long long to_fixed(double x, int E) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(x);
  int ex = (int)(u >> 52) & 0x7FF;
  unsigned long long m = u & 0xFFFFFFFFFFFFFull;
  if (ex)
    m |= 1ull << 52;
  else
    ex = 1;
  const int sh = ex - 1013 - E;   // <= 9
  unsigned long long r;
  if (sh >= 0) {
    r = m << sh;
  } else {
    const int k = -sh;
    r = k < 64 ? (m + (1ull << (k - 1))) >> k : 0ull;
  }
  return (u >> 63) ? -(long long)r : (long long)r;
}

// exponent of a row's largest magnitude from its bit pattern: 2^(E-1) <= max < 2^E
__device__ __forceinline__ int max_exp(unsigned long long mx) {
  const int ex = (int)(mx >> 52);
  if (ex == 0x7FF) return kBadExp;
  return (ex ? ex : 1) - 1022;
}
// x 2^-E (|x| < 2^E) in FP32, squared: a row's sum of these gives its norm to 1e-4
__device__ __forceinline__ float scaled_sq(double x, int E) {
  const float f = f64_to_f32(x, -E);
  return f * f;
}
// exponent of the row's 2-norm (an upper bound) from its maximum's and that sum
__device__ __forceinline__ int norm_exp(int E, float sq) {
  if (E == kBadExp) return E;
  const float s = sq * 1.001f;
  return s < 1.f ? E : E + (((int)(__float_as_uint(s) >> 23) - 127 + 2) >> 1);
}

// two integers |d| <= 512 as FP16 (1536 + d has unit spacing)
__device__ __forceinline__ unsigned pack_digits(int a, int b) {
  const unsigned u = (unsigned)(a + 512 + 0x6400) | ((unsigned)(b + 512 + 0x6400) << 16);
  const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&u), __half2half2(__float2half(1536.f)));
  return *reinterpret_cast<const unsigned*>(&h);
}

// the digit chunks (8 consecutive k) of eight fixed-point values
__device__ __forceinline__ void store_digits(long long* v, __half* dst, long long plane) {
#pragma unroll
  for (int s = NS - 1; s >= 0; --s) {
    int d[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (s > 0) {
        d[i] = (int)(signed char)(v[i] & 0xFF);
        v[i] = (v[i] + 128) >> 8;
      } else {
        d[i] = (int)v[i];
      }
    }
    uint4 q;
    q.x = pack_digits(d[0], d[1]);
    q.y = pack_digits(d[2], d[3]);
    q.z = pack_digits(d[4], d[5]);
    q.w = pack_digits(d[6], d[7]);
    *reinterpret_cast<uint4*>(dst + s * plane) = q;
  }
}

// halves offset of chunk j (k = 8j .. 8j + 7 of K block kb) of row r within a slab
__device__ __forceinline__ long long chunk_off(int rows_pad, int r, int kb, int j) {
  return ((long long)kb * rows_pad + r) * 32 + 8 * (j ^ ((r >> 1) & 3));
}
#endif

}  // namespace f64s

// exponents and digit planes of every form's rows
void launch_f64_slice(const f64s::SliceArgs& a, int nforms, cudaStream_t s);
// One persistent launch over the jobs' output tiles.  A bounded wait that gives up raises *err and
// leaves NaN in the tiles that its CTA has not finished, so that no call returns stale values.
int launch_f64_gemm(const f64s::Job* jobs, int njobs, int* err, cudaStream_t s, bool stall = false);

}  // namespace sbe
