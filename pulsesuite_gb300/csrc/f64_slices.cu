// Exact-slice FP64 products on tcgen05 (see f64_slices.cuh).
#include "f64_slices.cuh"
#include "fp_bits.cuh"
#include "per_device.cuh"
#include "sbe_internal.cuh"
#include "tc_ptx.cuh"

#include <algorithm>

namespace sbe {
namespace f64s {

// ---------------------------------------------------------------------------
// slicing

// Block: 8 rows, or with few K blocks (PACK) as many groups of 8 as its warps can take, of one
// form of one matrix; a group's warps (SPLIT: pairs of warps, real and imaginary
// part) walk the K blocks, a lane takes 8 consecutive k of one row (lane = 4 row + chunk), so a
// warp stores 512 contiguous bytes per plane and the transposed read covers 128-byte segments.  KB
// K blocks of a warp stay in registers between the row maximum, the norm and the digits (Nk up to
// 256 KB); longer rows are read again (from L2).  HBM bound: 16 B read and 32 B written per
// element.  The split halves a thread's chain of digits, which bounds a few small wires (1 x 64
// 8.9 -> 7.4 us a launch), and its registers, of which two K blocks take too many (2 x 512 75 ->
// 60); with one K block and many rows its 8-byte reads cost more (8 x 256 62 -> 70), and the warps
// that two K blocks leave idle take other rows (32 x 64 52 -> 27, 8 x 128 33 -> 28).
constexpr int kSliceStep = 8;   // K blocks in flight

// log2 of the warps that walk the K blocks of one group of 8 rows (PACK)
__host__ __device__ inline int slice_lgw(int nkb) { return nkb > 2 ? 2 : nkb - 1; }

template <int KB, bool SPLIT, bool PACK>
__global__ void __launch_bounds__(32 * kSliceStep * (SPLIT ? 2 : 1))
    k_f64_slice(const __grid_constant__ SliceArgs a) {
  pdl_enter();
  constexpr int kWarps = kSliceStep * (SPLIT ? 2 : 1), NC = SPLIT ? 1 : 2;
  const Form& f = a.f[blockIdx.y];
  const int kdim = a.kdim, ld = a.ld, b = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nkb = k_blocks(kdim), rows_pad = pad_rows(a.rows);
  const int im = SPLIT ? warp & 1 : 0, w = SPLIT ? warp >> 1 : warp;
  const int lgw = PACK ? slice_lgw(nkb) : 3, kStep = 1 << lgw, kw = w & (kStep - 1);
  const int g0 = PACK ? warp - kw : 0, gw = PACK ? kStep : kWarps;   // the group's warps
  const int r = ((blockIdx.x << (3 - lgw)) + (w >> lgw)) * 8 + (lane >> 2), j = lane & 3;
  const double2* X = f.src + (long long)b * a.src_batch;
  const double2* Y = f.add ? f.add + (long long)b * a.src_batch : nullptr;
  const bool rok = r < a.rows, held = nkb <= kStep * KB;
  auto load = [&](int kb, double (*v)[8]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int k = kb * BK + 8 * j + i;
      const long long o = f.transpose ? (long long)k * ld + r : (long long)r * ld + k;
      const bool in = rok && k < kdim && (k != r || !f.peel);
      if constexpr (SPLIT) {
        v[0][i] = in ? reinterpret_cast<const double*>(X)[2 * o + im] : 0.0;
        if (in && Y && im) v[0][i] += a.add_f * Y[(long long)r * ld + k].x;
      } else {
        const double2 z = in ? X[o] : make_double2(0.0, 0.0);
        v[0][i] = z.x;
        v[1][i] = z.y;
        if (in && Y) v[1][i] += a.add_f * Y[(long long)r * ld + k].x;
      }
    }
  };
  __shared__ unsigned long long red[kWarps][8];
  __shared__ float reds[kWarps][8];
  double v[KB][NC][8];
  unsigned long long m = 0;
  auto maximum = [&](const double (*x)[8]) {
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
      for (int i = 0; i < 8; ++i) m = max(m, absbits(x[c][i]));
  };
  if (held) {
#pragma unroll
    for (int u = 0; u < KB; ++u) load(kw + kStep * u, v[u]);   // zeros past the last K block
#pragma unroll
    for (int u = 0; u < KB; ++u) maximum(v[u]);
  } else {
    for (int kb = kw; kb < nkb; kb += kStep) {
      load(kb, v[0]);
      maximum(v[0]);
    }
  }
  m = max(m, __shfl_xor_sync(0xffffffffu, m, 1));
  m = max(m, __shfl_xor_sync(0xffffffffu, m, 2));
  if (j == 0) red[warp][lane >> 2] = m;
  __syncthreads();
  m = 0;
#pragma unroll
  for (int i = 0; i < kWarps; ++i)
    if (i < gw) m = max(m, red[g0 + i][lane >> 2]);
  const int Em = max_exp(m);
  float sq = 0.f;
  auto squares = [&](const double (*x)[8]) {
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
      for (int i = 0; i < 8; ++i) sq += scaled_sq(x[c][i], Em);
  };
  if (Em != kBadExp) {
    if (held) {
#pragma unroll
      for (int u = 0; u < KB; ++u) squares(v[u]);
    } else {
      for (int kb = kw; kb < nkb; kb += kStep) {
        load(kb, v[0]);
        squares(v[0]);
      }
    }
  }
  sq += __shfl_xor_sync(0xffffffffu, sq, 1);
  sq += __shfl_xor_sync(0xffffffffu, sq, 2);
  if (j == 0) reds[warp][lane >> 2] = sq;
  __syncthreads();
  sq = 0.f;
#pragma unroll
  for (int i = 0; i < kWarps; ++i)
    if (i < gw) sq += reds[g0 + i][lane >> 2];
  const int E = norm_exp(Em, sq);
  if (kw == 0 && im == 0 && j == 0 && rok) f.e[(long long)b * a.rows + r] = E;
  if (!rok) return;
  __half* dst = f.dst + (long long)b * a.dst_batch + im * NS * a.plane;
  auto digits = [&](int kb, const double (*x)[8]) {
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      long long q[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) q[i] = E == kBadExp ? 0 : to_fixed(x[c][i], E);
      store_digits(q, dst + chunk_off(rows_pad, r, kb, j) + c * NS * a.plane, a.plane);
    }
  };
  if (held) {
#pragma unroll
    for (int u = 0; u < KB; ++u)
      if (kw + kStep * u < nkb) digits(kw + kStep * u, v[u]);
  } else {
    for (int kb = kw; kb < nkb; kb += kStep) {
      load(kb, v[0]);
      digits(kb, v[0]);
    }
  }
}

// ---------------------------------------------------------------------------
// the product kernel

constexpr int A_SLICE = BM * BK * 2;       // 8 KB: one digit plane of an A tile
constexpr int A_GROUP = 4;                 // planes of a ring slot
constexpr int A_SLOT = A_GROUP * A_SLICE;  // 32 KB
constexpr int B_SLICE = BN * BK * 2;       // 4 KB
constexpr int B_SLOT = NS * B_SLICE;       // 32 KB: all planes of a B tile
constexpr int NA = 4, NB = 3;              // ring slots
constexpr int EPI_WARPS = 8;
constexpr int THREADS = 64 + 32 * EPI_WARPS;
constexpr int SMEM = 1024 + NA * A_SLOT + NB * B_SLOT + 512;

struct Unit {
  int job, b, m0, n0, comp, part;
  int kb0, nkb;     // K blocks of one real product
  int q0, q1;       // range of this part in the sequence of (product, K block)
  bool dead;
};

__device__ __forceinline__ Unit unit_of(const Launch& L, int u) {
  Unit t;
  int j = 0;
  while (j + 1 < L.njobs && L.base[j + 1] <= u) ++j;
  const Job& d = L.job[j];
  int r = u - L.base[j];
  const int tn = (d.N + BN - 1) / BN, tm = (d.M + BM - 1) / BM;
  t.job = j;
  t.n0 = (r % tn) * BN;
  r /= tn;
  t.m0 = (r % tm) * BM;
  r /= tm;
  t.comp = d.cplx ? r & 1 : 0;
  if (d.cplx) r >>= 1;
  t.part = r % d.parts;
  t.b = r / d.parts;
  t.kb0 = 0;
  t.nkb = d.nkb;
  t.dead = false;
  if (d.band) {
    // rows 2 dd + c of the sheared operand are zero outside t' in [-d, Nk - 1 - d], d =
    // dd - (Nk - 1); output (m, dd) is used only if m + dd lies in [Nk - 1, 2 Nk - 2]
    const int nk = d.band;
    const int dd_lo = t.n0 / 2, dd_hi = min((t.n0 + BN) / 2, 2 * nk - 1) - 1;
    const int tlo = max(0, nk - 1 - dd_hi), thi = min(nk - 1, 2 * nk - 2 - dd_lo);
    t.kb0 = tlo / BK;
    t.nkb = thi >= tlo ? thi / BK + 1 - t.kb0 : 0;
    const int m_hi = min(t.m0 + BM, d.M) - 1;
    t.dead = dd_lo + t.m0 > 2 * nk - 2 || dd_hi + m_hi < nk - 1;
  }
  const int n = t.nkb * (d.cplx ? 2 : 1);
  t.q0 = (int)((long long)t.part * n / d.parts);
  t.q1 = (int)((long long)(t.part + 1) * n / d.parts);
  return t;
}

// v 2^e rounded once to FP64, on the integer pipe while the result is normal
__device__ __forceinline__ double ll_scaled(long long v, int e) {
  if (v == 0) return 0.0;
  const unsigned long long sg = (unsigned long long)v & 0x8000000000000000ull;
  const unsigned long long a = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
  const int lz = __clzll((long long)a);
  const unsigned long long n = a << lz;
  const unsigned long long mant = (n >> 11) + ((n >> 10) & 1ull);   // 53 bits, half up
  const int ef = 1023 + 63 - lz + e;
  if (ef <= 0 || ef >= 2046) return ldexp((double)v, e);
  return __longlong_as_double((long long)(sg | (((unsigned long long)(ef - 1) << 52) + mant)));
}

__device__ __forceinline__ void st_global_v4(double* p, double a, double b, double c, double d) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a), "d"(b), "d"(c), "d"(d)
               : "memory");
}

// The accumulators of 16 of a thread's 32 columns into the running sums, in units of 2^6 of
// sum_t acc_t 2^(8 (7 - t)), modulo 2^64 (the whole sum stays below 2^62).  The conversion
// float -> int runs at an eighth of the FP32 rate, so every other accumulator takes a cheaper
// way: adding 1.5 2^25 leaves rint(a / 4) in the mantissa, and the remainder (at most 2, exact)
// goes to the next accumulator as 256 times itself, which keeps that below 2^24.  The bits are
// added with their offset; kBias per accumulation is taken off at the end.
constexpr float kMagic = 50331648.f;
constexpr uint32_t kMagicBits = 0x4C400000u;
__host__ __device__ constexpr int sum_shift(int t) { return 50 - 8 * t; }
constexpr unsigned long long kBias = ((unsigned long long)kMagicBits << (sum_shift(0) + 2)) +
                                     ((unsigned long long)kMagicBits << (sum_shift(2) + 2)) +
                                     ((unsigned long long)kMagicBits << (sum_shift(4) + 2));

template <int T>   // a: accumulator T, next: T + 1
__device__ __forceinline__ void add_magic(unsigned long long* run, const uint32_t* a, uint32_t* next) {
  constexpr int S = sum_shift(T) + 2;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const float v = __uint_as_float(a[j]), r = __fadd_rn(v, kMagic);
    const float e = __fsub_rn(v, __fsub_rn(r, kMagic));
    next[j] = __float_as_uint(__fmaf_rn(e, 256.f, __uint_as_float(next[j])));
    if constexpr (S >= 32)   // the high word alone changes
      run[j] += (unsigned long long)(__float_as_uint(r) << (S - 32)) << 32;
    else
      run[j] += (unsigned long long)__float_as_uint(r) * (1u << S);
  }
}
template <int T>
__device__ __forceinline__ void add_acc(unsigned long long* run, const uint32_t* a) {
  constexpr int S = sum_shift(T);
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const int v = __float2int_rn(__uint_as_float(a[j]));
    if constexpr (S >= 32)
      run[j] += (unsigned long long)((unsigned)v << (S - 32)) << 32;
    else
      run[j] += (unsigned long long)((long long)v * (1 << S));
  }
}
// accumulators 6 and 7 (rounded to two units at most)
__device__ __forceinline__ void add_acc67(unsigned long long* run, const uint32_t* a6,
                                          const uint32_t* a7) {
#pragma unroll
  for (int j = 0; j < 16; ++j)
    run[j] += (unsigned long long)(long long)__float2int_rn(
        fmaf(__uint_as_float(a7[j]), 1.f / 64.f, __uint_as_float(a6[j]) * 4.f));
}

// Persistent, one CTA per SM: warp 0 streams digit planes (bulk copies; A planes in groups of
// four, B tiles whole), warp 1 issues the MMAs, warps 2-9 drain the accumulators.  A tile is
// 128 x 64: its eight accumulators fill the 512 TMEM columns at 64 t, so the plane A_i against
// adjacent planes of B (rows adjacent in shared memory) is one MMA of N up to 256 onto adjacent
// accumulators: 36 plane products per K block in 12 MMAs per 16 k.  The accumulators are
// drained every 128 k (exactness).  They form two windows, t >= 4 (26 of the 36 products) and
// t < 4, each with its own barriers: the epilogue drains the upper window while the last MMAs of
// the lower run, and the lower while the next upper ones do.
// 1 wire x Nk = 512, the twelve commutator products (464 GFLOP of MMA work): 617 us with a
// barrier per plane (the issuing thread's waits), 448 with grouped ones, 417 with the windows and
// fewer conversions, 340 with the drain in 16-column steps (no spills) and 32-byte stores, of
// which the MMAs alone take 304.
__global__ void __launch_bounds__(THREADS, 1) k_f64_gemm(const __grid_constant__ Launch L) {
  pdl_enter();
  using namespace tc;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~uintptr_t(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + NA * A_SLOT;
  uint64_t* fullA = reinterpret_cast<uint64_t*>(sB + NB * B_SLOT);
  uint64_t* emptyA = fullA + NA;
  uint64_t* fullB = emptyA + NA;
  uint64_t* emptyB = fullB + NB;
  uint64_t* tfull = emptyB + NB;    // per window: 0 lower (t < 4), 1 upper
  uint64_t* tempty = tfull + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x / 32, lane = threadIdx.x & 31;
  const int nunits = L.base[L.njobs];
  int* err = L.err;
  if (threadIdx.x == 0) {
    for (int i = 0; i < NA; ++i) {
      mbar_init(&fullA[i], 1);
      mbar_init(&emptyA[i], 1);
    }
    for (int i = 0; i < NB; ++i) {
      mbar_init(&fullB[i], 1);
      mbar_init(&emptyB[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull[i], 1);
      mbar_init(&tempty[i], EPI_WARPS);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0 && lane == 0) {
    // ---------------- producer ----------------
    int sa = 0, sb = 0;
    uint32_t pa = 0, pb = 0;   // phases of the ring positions
    long long na = 0, nb = 0;
    bool ok = true;
    for (int u = blockIdx.x; ok && !L.stall && u < nunits; u += gridDim.x) {
      const Unit t = unit_of(L, u);
      if (t.dead) continue;
      const Job& d = L.job[t.job];
      for (int q = t.q0; ok && q < t.q1; ++q) {
        const int p = q >= t.nkb ? 1 : 0, kb = t.kb0 + q - p * t.nkb;
        // re: Ar Br, Ai Bi; im: Ar Bi, Ai Br
        const int ca = p, cb = t.comp ? 1 - p : p;
        const __half* gb = d.B + (long long)cb * NS * d.b_plane + (long long)t.b * d.b_batch +
                           ((long long)kb * d.b_pad + t.n0) * BK;
        if (!mbar_wait(&emptyB[sb], pb ^ 1u, err, abort_flag)) {
          ok = false;
          break;
        }
        mbar_expect_tx(&fullB[sb], B_SLOT);
        for (int i = 0; i < NS; ++i)
          bulk_load(sB + sb * B_SLOT + i * B_SLICE, gb + i * d.b_plane, B_SLICE, &fullB[sb]);
        ++nb;
        if (++sb == NB) {
          sb = 0;
          pb ^= 1u;
        }
        const __half* ga = d.A + (long long)ca * NS * d.a_plane + (long long)t.b * d.a_batch +
                           ((long long)kb * d.a_pad + t.m0) * BK;
        for (int i = 0; i < NS; i += A_GROUP) {
          if (!mbar_wait(&emptyA[sa], pa ^ 1u, err, abort_flag)) {
            ok = false;
            break;
          }
          mbar_expect_tx(&fullA[sa], A_SLOT);
          for (int j = 0; j < A_GROUP; ++j)
            bulk_load(sA + sa * A_SLOT + j * A_SLICE, ga + (i + j) * d.a_plane, A_SLICE,
                      &fullA[sa]);
          ++na;
          if (++sa == NA) {
            sa = 0;
            pa ^= 1u;
          }
        }
      }
    }
    // no copy may land in shared memory after the CTA has gone: wait (bounded) for the
    // last ones issued
    volatile int never = 0;
    for (long long i = na > NA ? na - NA : 0; i < na; ++i)
      mbar_wait(&fullA[i % NA], (uint32_t)((i / NA) & 1), err, &never);
    for (long long i = nb > NB ? nb - NB : 0; i < nb; ++i)
      mbar_wait(&fullB[i % NB], (uint32_t)((i / NB) & 1), err, &never);
  } else if (warp == 1 && lane == 0) {
    // ---------------- MMA issuer ----------------
    int sa = 0, sb = 0;
    uint32_t pa = 0, pb = 0, pt = 1;   // tempty: the first wait passes at once
    bool ok = true;
    for (int u = blockIdx.x; ok && u < nunits; u += gridDim.x) {
      const Unit t = unit_of(L, u);
      if (t.dead) continue;
      const Job& d = L.job[t.job];
      // signs of the two real products: re = Ar Br - Ai Bi, im = Ar Bi + Ai Br with the
      // conjugations' signs on the imaginary planes
      const int s0 = t.comp ? (d.conj_b ? -1 : 1) : 1;
      const int s1 = t.comp ? (d.conj_a ? -1 : 1) : -(d.conj_a ? -1 : 1) * (d.conj_b ? -1 : 1);
      for (int c0 = t.q0; ok && c0 < t.q1; c0 += CHUNK) {
        const int c1 = min(c0 + CHUNK, t.q1);
        for (int q = c0; q < c1; ++q) {
          const int sg = (q >= t.nkb ? s1 : s0) * (d.neg ? -1 : 1);
          const uint32_t id = idesc_f16(BM, 0, sg < 0 ? 1 : 0);
          const uint32_t first = q == c0 ? 0u : 1u;
          const int sa1 = sa + 1;   // NA is even: the groups of a K block are adjacent slots
          if (!mbar_wait(&fullB[sb], pb, err, abort_flag) ||
              !mbar_wait(&fullA[sa], pa, err, abort_flag) ||
              !mbar_wait(&fullA[sa1], pa, err, abort_flag) ||
              (q == c0 && !mbar_wait(&tempty[1], pt, err, abort_flag))) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint64_t da = sw64_desc(smem_u32(sA + sa * A_SLOT));
          const uint64_t db = sw64_desc(smem_u32(sB + sb * B_SLOT));
          // upper window: A_i with B_{max(0, 4 - i)} .. B_{7 - i} onto accumulators max(4, i) .. 7
#pragma unroll
          for (int i = 0; i < NS; ++i) {
            const int j0 = i < 4 ? 4 - i : 0, t0 = i < 4 ? 4 : i, n = 8 - t0;
#pragma unroll
            for (int k16 = 0; k16 < 2; ++k16)
              umma_f16(tmem + t0 * BN, da + (uint64_t)(i * (A_SLICE >> 4) + 2 * k16),
                       db + (uint64_t)(j0 * (B_SLICE >> 4) + 2 * k16),
                       id + ((uint32_t)(n * BN >> 3) << 17), (i == 0 && k16 == 0) ? first : 1u);
          }
          umma_commit(&emptyA[sa1]);
          if (q == c1 - 1) umma_commit(&tfull[1]);
          if (q == c0) {
            if (!mbar_wait(&tempty[0], pt, err, abort_flag)) {
              ok = false;
              break;
            }
            tc_fence_after();
          }
          // lower window: A_i with B_0 .. B_{3 - i} onto accumulators i .. 3
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int k16 = 0; k16 < 2; ++k16)
              umma_f16(tmem + i * BN, da + (uint64_t)(i * (A_SLICE >> 4) + 2 * k16),
                       db + 2u * k16, id + ((uint32_t)((4 - i) * BN >> 3) << 17),
                       (i == 0 && k16 == 0) ? first : 1u);
          umma_commit(&emptyA[sa]);
          umma_commit(&emptyB[sb]);
          sa += 2;
          if (sa == NA) {
            sa = 0;
            pa ^= 1u;
          }
          if (++sb == NB) {
            sb = 0;
            pb ^= 1u;
          }
        }
        pt ^= 1u;
        if (ok) umma_commit(&tfull[0]);
      }
    }
  } else if (warp >= 2) {
    // ---------------- epilogue: 32 columns of one row per thread ----------------
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const uint32_t ta = tmem + ((uint32_t)(32 * quarter) << 16) + half * 32;
    uint32_t pt = 0;
    bool ok = true;   // after a wait that gave up the tiles left become NaN
    for (int u = blockIdx.x; u < nunits; u += gridDim.x) {
      const Unit t = unit_of(L, u);
      if (t.dead) continue;
      const Job& d = L.job[t.job];
      unsigned long long run[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) run[j] = 0;
      unsigned long long bias = 0;
      for (int c0 = t.q0; ok && c0 < t.q1; c0 += CHUNK) {
        uint32_t a[16], b[16];
        if (!mbar_wait(&tfull[1], pt, err, abort_flag)) {
          ok = false;
          break;
        }
        tc_fence_after();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          tmem_ld16_nw(ta + 4 * BN + 16 * h, a);
          tmem_ld16_nw(ta + 5 * BN + 16 * h, b);
          tmem_ld_wait();
          add_magic<4>(run + 16 * h, a, b);
          add_acc<5>(run + 16 * h, b);
          tmem_ld16_nw(ta + 6 * BN + 16 * h, a);
          tmem_ld16_nw(ta + 7 * BN + 16 * h, b);
          tmem_ld_wait();
          if (h == 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tempty[1]);
          }
          add_acc67(run + 16 * h, a, b);
        }
        if (!mbar_wait(&tfull[0], pt, err, abort_flag)) {
          ok = false;
          break;
        }
        pt ^= 1u;
        tc_fence_after();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          tmem_ld16_nw(ta + 16 * h, a);
          tmem_ld16_nw(ta + 1 * BN + 16 * h, b);
          tmem_ld_wait();
          add_magic<0>(run + 16 * h, a, b);
          add_acc<1>(run + 16 * h, b);
          tmem_ld16_nw(ta + 2 * BN + 16 * h, a);
          tmem_ld16_nw(ta + 3 * BN + 16 * h, b);
          tmem_ld_wait();
          if (h == 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tempty[0]);
          }
          add_magic<2>(run + 16 * h, a, b);
          add_acc<3>(run + 16 * h, b);
        }
        bias += kBias;
      }
      const int m = t.m0 + 32 * quarter + lane;
      if (m >= d.M) continue;
      const int ea = ok ? d.ea[(long long)t.b * d.M + m] : kBadExp;
      const int* eb = d.eb + (long long)t.b * d.N;
      double* o = d.out + t.part * d.o_part + t.comp * d.o_comp + (long long)t.b * d.o_batch;
      const int n0 = t.n0 + 32 * half;
      if (d.band) {
        // column 2 dd + c of row m: component c of element [m][m + dd - (Nk - 1)]
        const int nk = d.band;
        o += (long long)m * d.ldo;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const int n = n0 + j, k2 = m + (n >> 1) - (nk - 1);
          if (n < d.N && k2 >= 0 && k2 < nk) {
            const int e = eb[n];
            o[2 * k2 + (n & 1)] = (ea == kBadExp || e == kBadExp)
                                      ? __longlong_as_double(0x7FF8000000000000ll)
                                      : ll_scaled((long long)(run[j] - bias), ea + e - 62);
          }
        }
      } else {
        o += (long long)m * d.ldo + n0;
        auto value = [&](int j) {
          const int e = eb[n0 + j];
          return (ea == kBadExp || e == kBadExp) ? __longlong_as_double(0x7FF8000000000000ll)
                                                 : ll_scaled((long long)(run[j] - bias), ea + e - 62);
        };
        // a thread's 32 columns are 256 contiguous bytes: 32-byte stores where rows allow
        if ((d.ldo & 3) == 0 && n0 + 32 <= d.N) {
#pragma unroll
          for (int j = 0; j < 32; j += 4)
            st_global_v4(o + j, value(j), value(j + 1), value(j + 2), value(j + 3));
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (n0 + j < d.N) o[j] = value(j);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

}  // namespace f64s

void launch_f64_slice(const f64s::SliceArgs& a, int nforms, cudaStream_t s) {
  const int nkb = f64s::k_blocks(a.kdim);
  dim3 grid((a.rows + 7) / 8, nforms, a.batch);
  const long long blocks = (long long)grid.x * grid.y * grid.z;
  if (nkb > f64s::kSliceStep) {
    launch(f64s::k_f64_slice<2, true, false>, grid, 512, 0, s, a);
  } else if (blocks < 4 * 152) {
    launch(f64s::k_f64_slice<1, true, false>, grid, 512, 0, s, a);
  } else if (nkb > 4) {
    launch(f64s::k_f64_slice<1, false, false>, grid, 256, 0, s, a);
  } else {
    const int per = 8 << (3 - f64s::slice_lgw(nkb));
    grid.x = (a.rows + per - 1) / per;
    launch(f64s::k_f64_slice<1, false, true>, grid, 256, 0, s, a);
  }
}

int launch_f64_gemm(const f64s::Job* jobs, int njobs, int* err, cudaStream_t s, bool stall) {
  if (njobs < 1 || njobs > f64s::MAX_JOBS) return fail(SBE_ERR_ARG, "f64 gemm: 1 to 16 jobs");
  const int rc = cuda_check(raise_smem<f64s::k_f64_gemm>(f64s::SMEM), "f64 gemm: shared-memory limit");
  if (rc) return rc;
  f64s::Launch L{};
  L.njobs = njobs;
  L.err = err;
  L.stall = stall;
  long long nt = 0;
  for (int j = 0; j < njobs; ++j) {
    const f64s::Job& d = jobs[j];
    if (d.M < 1 || d.N < 1 || d.nkb < 1 || d.batch < 1 || d.parts < 1 || d.a_pad % 128 ||
        d.b_pad % 64 || d.M > d.a_pad || d.N > d.b_pad)
      return fail(SBE_ERR_ARG, "f64 gemm: bad job");
    L.job[j] = d;
    L.base[j] = (int)nt;
    nt += (long long)((d.N + f64s::BN - 1) / f64s::BN) * ((d.M + f64s::BM - 1) / f64s::BM) *
          (d.cplx ? 2 : 1) * d.parts * d.batch;
  }
  if (nt > 0x7FFFFFFF) return fail(SBE_ERR_ARG, "f64 gemm: too many tiles");
  L.base[njobs] = (int)nt;
  const int grid = (int)std::min<long long>(nt, sm_count());
  launch(f64s::k_f64_gemm, grid, f64s::THREADS, f64s::SMEM, s, L);
  return cuda_check(cudaGetLastError(), "f64 gemm launch");
}

int f64_wait_selftest(double* out, int* err, cudaStream_t s) {
  int* e = nullptr;   // row exponents, and the operands that nothing reads
  if (cudaMallocAsync(&e, 256, s) != cudaSuccess)
    return fail(SBE_ERR_OOM, "sbe_f64_wait_selftest: scratch allocation failed");
  cudaMemsetAsync(e, 0, 256, s);
  f64s::Job j{};
  j.A = j.B = reinterpret_cast<const __half*>(e);
  j.a_pad = j.b_pad = 128;
  j.ea = j.eb = e;
  j.M = j.N = j.ldo = 64;
  j.nkb = 2;
  j.batch = j.parts = 1;
  j.out = out;
  const int rc = launch_f64_gemm(&j, 1, err, s, true);
  cudaFreeAsync(e, s);
  return rc;
}

}  // namespace sbe
