// The FP64 right-hand side on exact-slice tensor-core products (f64_slices.cuh): exchange
// sums, commutators and sources of the FP64 path, per bucket of wires of one Nk.
#include <algorithm>
#include <map>
#include <mutex>
#include <vector>

#include "f64_slices.cuh"
#include "sbe_ctx.cuh"

namespace sbe {

using f64s::BK;
using f64s::chunk_off;
using f64s::k_blocks;
using f64s::kBadExp;
using f64s::NS;
using f64s::pad_rows;
using f64s::max_exp;
using f64s::norm_exp;
using f64s::scaled_sq;
using f64s::store_digits;
using f64s::to_fixed;

// operand forms (rows as stored, or transposed)
enum { F_P = 0, F_PT, F_C, F_CT, F_D, F_DT, F_EH, F_EHT, F_EE, F_EET, F_HH, F_HHT, F_EEX, F_HHX, F_N };

// The commutators' forms of C, D, Hee and Hhh leave the diagonal (occupations and band energies)
// to the finish, which applies it element by element in FP64: a row held in fixed point under a
// norm that its diagonal element sets would keep a coherence of 1e-8 of it to 1e-9 only.
static int peeled(int f) { return f != F_P && f != F_PT && f != F_EH && f != F_EHT; }

struct F64Bucket {
  int nk = 0, nw = 0, nr = 0, group = 0;   // group: wires per pass
  long long bm = 0, bv = 0, br = 0, bkr = 0;
  WireDev* dw = nullptr;
  void* block = nullptr;
  __half *pl = nullptr, *sp = nullptr, *tp = nullptr, *ep = nullptr;
  int *ef = nullptr, *es = nullptr, *et = nullptr, *ee = nullptr;
  double *xsh = nullptr, *part = nullptr;
  int parts = 1, sparts = 1;   // cuts of the commutator and source products
  long long sl_m = 0, sl_s = 0, sl_e = 0;   // slabs: Nk x Nk, sheared, E^T
};
struct F64Work {
  std::vector<F64Bucket> b;
};

static F64Work* work_of(SbeCtx* c) { return static_cast<F64Work*>(c->f64); }

void f64_free(SbeCtx* c) {
  F64Work* w = work_of(c);
  if (!w) return;
  for (auto& b : w->b) {
    cudaFree(b.block);
    cudaFree(b.dw);
  }
  delete w;
  c->f64 = nullptr;
}

// ---------------------------------------------------------------------------
// Diagonals of P, C, D: the sums of C and D (the traces of the direct Coulomb terms,
// SBEs.py:1094-1103; layout and order of k_traces) and the norm's exponent, that
// of the sheared rows 2 dd, 2 dd + 1 (dd = row - column + Nk - 1).  One warp per diagonal.
__global__ void __launch_bounds__(128) k_f64_diag(int nk, const double2* P, const double2* C,
                                                  const double2* D, double2* tr, int* es) {
  pdl_enter();
  const int i = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (i >= 2 * nk - 1) return;
  const int d = i - (nk - 1), which = blockIdx.y, b = blockIdx.z;   // column - row
  const double2* X = (which == 0 ? P : which == 1 ? C : D) + (long long)b * nk * nk;
  const int k0 = d >= 0 ? 0 : -d, k1 = d >= 0 ? nk - 1 - d : nk - 1;
  double sr = 0.0, si = 0.0;
  unsigned long long m = 0;
  for (int k = k0 + lane; k <= k1; k += 32) {
    const double2 v = X[(long long)k * nk + k + d];
    sr += v.x;
    si += v.y;
    m = max(m, max(absbits(v.x), absbits(v.y)));
  }
  for (int o = 16; o > 0; o >>= 1) {
    sr += __shfl_down_sync(0xffffffffu, sr, o);
    si += __shfl_down_sync(0xffffffffu, si, o);
    m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  }
  const int Em = max_exp(m);
  float sq = 0.f;
  if (Em != kBadExp)
    for (int k = k0 + lane; k <= k1; k += 32) {
      const double2 v = X[(long long)k * nk + k + d];
      sq += scaled_sq(v.x, Em) + scaled_sq(v.y, Em);
    }
  for (int o = 16; o > 0; o >>= 1) sq += __shfl_down_sync(0xffffffffu, sq, o);
  if (lane == 0) {
    if (which > 0) tr[(long long)b * 4 * nk + (which - 1) * 2 * nk + d + nk] = make_double2(sr, si);
    if (es) {
      const int E = norm_exp(Em, sq);
      int* e = es + ((long long)which * gridDim.z + b) * (4 * nk - 2) + 2 * (nk - 1 - d);
      e[0] = E;
      e[1] = E;
    }
  }
}

__host__ __device__ inline int shear_first(int nk, int t0) {
  const int lo = nk - 63 - t0;   // lowest dd whose source rows can reach row 0
  return lo > 0 ? lo / 32 : 0;
}
__host__ __device__ inline bool shear_live(int nk, int t0, int dd0) {
  const int rb = t0 + dd0 - (nk - 1);
  return rb + 62 >= 0 && rb < nk;
}

// Digit planes of the sheared states: row 2 dd + c, column t' holds component c of
// X[t' + d][t'], d = dd - (Nk - 1).  A block takes 32 dd x 32 t' from a 63 x 32 tile read
// row by row; the blocks outside the band are never written (the planes start as zeros).
__global__ void __launch_bounds__(256) k_f64_shear(int nk, int nw, const double2* P,
                                                   const double2* C, const double2* D,
                                                   const int* es, __half* dst, long long slab) {
  pdl_enter();
  __shared__ double2 tile[63][33];
  const int n = blockIdx.z / nw, b = blockIdx.z % nw;
  const int t0 = blockIdx.x * 32, dd0 = (shear_first(nk, t0) + blockIdx.y) * 32;
  if (dd0 >= 2 * nk || !shear_live(nk, t0, dd0)) return;
  const double2* X = (n == 0 ? P : n == 1 ? C : D) + (long long)b * nk * nk;
  const int rb = t0 + dd0 - (nk - 1), tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int rr = ty + 8 * k, r = rb + rr, col = t0 + tx;
    if (rr < 63)
      tile[rr][tx] = (r >= 0 && r < nk && col < nk) ? X[(long long)r * nk + col]
                                                   : make_double2(0.0, 0.0);
  }
  __syncthreads();
  const int rl = ty * 8 + (tx >> 2), j = tx & 3, ddl = rl >> 1, row = 2 * dd0 + rl;
  const int E = row < 4 * nk - 2 ? es[((long long)n * nw + b) * (4 * nk - 2) + row] : kBadExp;
  long long q[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const double2 v = tile[8 * j + i + ddl][8 * j + i];
    q[i] = E == kBadExp ? 0 : to_fixed((rl & 1) ? v.y : v.x, E);
  }
  store_digits(q, dst + ((long long)n * NS * nw + b) * slab +
                      chunk_off(pad_rows(4 * nk), row, t0 >> 5, j),
               (long long)nw * slab);
}

// Digit planes of the Toeplitz operands T_n[t][t'] = v_n(|t - t'|), zero diagonal (n = eh,
// ee, hh), with one exponent per wire and n.  vs: 3 x Nk per wire (by |t - t'|).
__global__ void __launch_bounds__(256) k_f64_toeplitz(int nk, int nw, const double* vs, __half* dst,
                                                      int* et, long long slab) {
  pdl_enter();
  const int n = blockIdx.y, b = blockIdx.z, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const double* v = vs + ((long long)b * 3 + n) * nk;
  __shared__ unsigned long long red[8];
  __shared__ float reds[8];
  unsigned long long m = 0;
  for (int i = 1 + threadIdx.x; i < nk; i += 256) m = max(m, absbits(v[i]));
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) red[warp] = m;
  __syncthreads();
  m = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) m = max(m, red[w]);
  const int Em = max_exp(m);
  float sq = 0.f;
  if (Em != kBadExp)   // every off-diagonal value at most twice per row
    for (int i = 1 + threadIdx.x; i < nk; i += 256) sq += 2.f * scaled_sq(v[i], Em);
  for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
  if (lane == 0) reds[warp] = sq;
  __syncthreads();
  sq = 0.f;
#pragma unroll
  for (int w = 0; w < 8; ++w) sq += reds[w];
  const int E = norm_exp(Em, sq);
  const int r = blockIdx.x * 8 + (lane >> 2), j = lane & 3;
  if (r >= nk) return;
  if (warp == 0 && j == 0) et[((long long)n * nw + b) * nk + r] = E;
  __half* d = dst + ((long long)n * NS * nw + b) * slab;
  for (int kb = warp; kb < k_blocks(nk); kb += 8) {
    long long q[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int k = kb * BK + 8 * j + i, a = k > r ? k - r : r - k;
      q[i] = (E == kBadExp || a == 0 || k >= nk) ? 0 : to_fixed(v[a], E);
    }
    store_digits(q, d + chunk_off(pad_rows(nk), r, kb, j), (long long)nw * slab);
  }
}

// ---------------------------------------------------------------------------
// SBEs.py:1044-1131 and 5153-5163 from the exchange sums xsh[n][b][k1][k2] (n = P, C, D):
// the Hamiltonians of the wires, as calch_point forms them.
struct HBuild {
  int nk, nr, nw;
  const WireDev* wires;            // null: the single-wire call
  const double2 *C, *D, *Ek;       // C, D: diagonals without LF
  const double *vs, *Ee, *Eh;
  const double2 *tr, *xsh;
  const double2 *Meh, *Wee, *Whh;  // single-wire call
  double gap;
  int excitons, lf, freepot;
  double2 *Heh, *Hee, *Hhh;
};

__global__ void __launch_bounds__(128) k_f64_hbuild(const __grid_constant__ HBuild a) {
  pdl_enter();
  const int nk = a.nk, k2 = blockIdx.x * 128 + threadIdx.x, k1 = blockIdx.y, b = blockIdx.z;
  if (k2 >= nk) return;
  const long long mb = (long long)b * nk * nk, o = (long long)k1 * nk + k2;
  bool exc = a.excitons, lf = a.lf;
  double gap = a.gap;
  double2 heh = make_double2(0.0, 0.0);
  if (a.wires) {
    const WireDev& W = a.wires[b];
    exc = (W.flags & SBE_F_EXCITONS) != 0;
    lf = (W.flags & SBE_F_LF) != 0;
    gap = W.gap;
    if (a.Ek && (W.flags & SBE_F_OPTICS)) {
      int q = k1 - k2;
      if (q < 0) q += a.nr;
      const double2* ek = a.Ek + (long long)b * 3 * a.nr;
      const double2 ex = ek[q], ey = ek[a.nr + q], ez = ek[2 * a.nr + q];
      const double xcv = W.dcv * ((k2 & 1) ? -1.0 : 1.0);
      const double2 t1 = cscale(ex, -W.ehint * xcv);
      const double2 t2 = cscale(cscale(ey, W.ehint * W.dcv), (double)W.yw);
      const double2 t3 = cscale(cscale(ez, W.ehint * -W.dcv), (double)W.zsign);
      heh = csub(csub(t1, t2), t3);
    }
  } else {
    heh = a.Meh[o];
  }
  double2 hee = make_double2(0.0, 0.0), hhh = hee;
  if (k1 == k2) {
    hee.x = a.Ee[(long long)b * nk + k1] + gap;
    hhh.x = a.Eh[(long long)b * nk + k1];
  }
  if (a.freepot) {
    hee = cadd(hee, a.Wee[o]);
    hhh = cadd(hhh, a.Whh[o]);
  }
  if (exc) {
    const long long pl = (long long)a.nw * nk * nk;
    const double2* x = a.xsh + mb + o;
    heh = cadd(heh, x[0]);
    const double *v0 = a.vs + 3ll * b * nk, *v1 = v0 + nk, *v2 = v1 + nk;
    if (lf) {
      hee = csub(hee, x[pl]);
      hhh = csub(hhh, x[2 * pl]);
      const int d = k1 - k2;
      if (d != 0) {
        const int ad = d < 0 ? -d : d;
        const double2* t = a.tr + 4ll * b * nk;
        const double2 trC = t[d + nk], trCm = t[-d + nk];
        const double2 trD = t[2 * nk + d + nk], trDm = t[2 * nk - d + nk];
        hee.x += v1[ad] * trC.x - v0[ad] * trDm.x;
        hee.y += v1[ad] * trC.y - v0[ad] * trDm.y;
        hhh.x += v2[ad] * trD.x - v0[ad] * trCm.x;
        hhh.y += v2[ad] * trD.y - v0[ad] * trCm.y;
      }
    } else if (k1 == k2) {
      for (int j = 0; j < nk; ++j) {
        if (j == k1) continue;
        const int aq = j < k1 ? k1 - j : j - k1;
        const double2 cv = a.C[mb + (long long)j * nk + j], dv = a.D[mb + (long long)j * nk + j];
        hee.x -= v1[aq] * cv.x;
        hee.y -= v1[aq] * cv.y;
        hhh.x -= v2[aq] * dv.x;
        hhh.y -= v2[aq] * dv.y;
      }
    }
  }
  a.Heh[mb + o] = heh;
  a.Hee[mb + o] = hee;
  a.Hhh[mb + o] = hhh;
}

// dP, dC, dD from the partial products (SBEs.py:1942-1965, 2309-2327, 2607-2625): the sum
// of each output's partials and of the terms with a diagonal element of C, D, Hee, Hhh,
//   dP: P_mn (Hhh_mm + Hee_nn) + Heh_nm (1 - D_mm - C_nn)
//   dC: Hee_nm (C_mm - C_nn) + C_mn (Hee_nn - Hee_mm),   dD with Hhh and D,
// over i hbar (dP's with the Heh^T of its own), for dP also the rates and OffP; with stage 1-4 the RK4 update of
// k_rk4_axpy.  Bound by the FP64 pipes (some 45 operations an element); one element a thread, so
// that a few small wires reach all SMs (four elements a thread: 1 x 64 13.3 us, 2 x 512 93; one: 4.7
// and 81).  The diagonals' terms take it from 81 to 112 us at 2 x 512, 56 to 87 at 8 x 256, 4.7 to
// 5.2 at 1 x 64.
struct Finish {
  int nk, nw, nsum, stage, first;   // first: output of blockIdx.z / nw = 0 (single calls)
  double dt, dt6;                   // the step, and a sixth of it
  const double* part;               // [output][nsum][re, im][wire][Nk x Nk]
  const double2 *X0[3], *H[3];      // P, C, D and Heh, Hee, Hhh
  const double2* offp;
  const double *gamE, *gamH;
  double2 *out[3], *X[3], *acc[3], *xs[3];
};

__global__ void __launch_bounds__(256) k_f64_finish(const __grid_constant__ Finish a) {
  pdl_enter();
  __shared__ double2 ht[32][9], dn[2][32], dm[2][8];
  const int nk = a.nk, which = blockIdx.z / a.nw + a.first, b = blockIdx.z % a.nw;
  const int m0 = blockIdx.y * 8, n0 = blockIdx.x * 32, tx = threadIdx.x, ty = threadIdx.y;
  const long long mm = (long long)nk * nk, mb = (long long)b * mm;
  {
    // the output's Hamiltonian transposed, and the diagonals: energies (0) and occupations (1) that
    // go with column n and with row m (dP: Hee, C and Hhh, D)
    const int t = ty * 32 + tx, n = n0 + (t >> 3), m = m0 + (t & 7);
    if (n < nk && m < nk) ht[t >> 3][t & 7] = a.H[which][mb + (long long)n * nk + m];
    const int kn = which == 2 ? 2 : 1, km = which == 1 ? 1 : 2;
    if (ty < 2 && n0 + tx < nk)
      dn[ty][tx] = (ty ? a.X0 : a.H)[kn][mb + (long long)(n0 + tx) * (nk + 1)];
    else if (ty < 4 && ty >= 2 && tx < 8 && m0 + tx < nk)
      dm[ty - 2][tx] = (ty == 3 ? a.X0 : a.H)[km][mb + (long long)(m0 + tx) * (nk + 1)];
    __syncthreads();
  }
  const double ih = 1.0 / kHbar;
  const long long cs = (long long)a.nw * mm;
  const double* part = a.part + (long long)(which - a.first) * a.nsum * 2 * cs + mb;
  const int m = m0 + ty, n = n0 + tx;
  if (m >= nk || n >= nk) return;
  const long long o = (long long)m * nk + n;
  const long long i = mb + o;
  double2 x0 = make_double2(0.0, 0.0), s0 = x0;
  if (a.stage > 0) x0 = a.X[which][i];
  if (a.stage > 1) s0 = a.acc[which][i];
  const double2 x = a.X0[which][i];
  double sx = 0.0, sy = 0.0;
  for (int s = 0; s < a.nsum; s += 4) {   // a multiple of four: eight loads in flight
    double p[4], q[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      p[u] = part[2 * (s + u) * cs + o];
      q[u] = part[(2 * (s + u) + 1) * cs + o];
    }
    const double tp = (p[0] + p[1]) + (p[2] + p[3]), tq = (q[0] + q[1]) + (q[2] + q[3]);
    sx = s ? sx + tp : tp;
    sy = s ? sy + tq : tq;
  }
  const double2 h = ht[tx][ty];
  {
    // x (e_n - e_m) + h (w_m - w_n), for dP x (e_n + e_m) + h (1 - w_m - w_n)
    const double2 en = dn[0][tx], wn = dn[1][tx], em = dm[0][ty], wm = dm[1][ty];
    double2 e, w;
    if (which == 0) {
      e = cadd(en, em);
      w = make_double2(1.0 - (wm.x + wn.x), -(wm.y + wn.y));
    } else {
      e = csub(en, em);
      w = csub(wm, wn);
    }
    sx = fma(x.x, e.x, fma(-x.y, e.y, fma(h.x, w.x, fma(-h.y, w.y, sx))));
    sy = fma(x.x, e.y, fma(x.y, e.x, fma(h.x, w.y, fma(h.y, w.x, sy))));
  }
  double2 v = make_double2(sy * ih, -sx * ih);
  if (which == 0) {
    const double gam = a.gamE[(long long)b * nk + n] + a.gamH[(long long)b * nk + m];
    v.x -= gam * x.x;
    v.y -= gam * x.y;
    if (a.offp) {
      const double2 f = a.offp[mb + o];
      v.x += f.y * ih;
      v.y += -f.x * ih;
    }
  }
  if (a.stage == 0) {
    a.out[which][i] = v;
  } else if (a.stage == 1) {
    a.acc[which][i] = v;
    a.xs[which][i] = make_double2(x0.x + 0.5 * a.dt * v.x, x0.y + 0.5 * a.dt * v.y);
  } else if (a.stage < 4) {
    a.acc[which][i] = make_double2(s0.x + 2.0 * v.x, s0.y + 2.0 * v.y);
    const double f = a.stage == 2 ? 0.5 * a.dt : a.dt;
    a.xs[which][i] = make_double2(x0.x + f * v.x, x0.y + f * v.y);
  } else {
    a.X[which][i] = make_double2(x0.x + a.dt6 * (s0.x + v.x), x0.y + a.dt6 * (s0.y + v.y));
  }
}

// ---------------------------------------------------------------------------
// products

// Terms of the three outputs: A form, B^T form, conjugations, sign.
struct TermDef {
  int a, b, ca, cb, neg;
};
static const TermDef kTerms[3][4] = {
    // Hhh P - D^T Heh^T + P Hee^T - Heh^T C
    {{F_HHX, F_PT, 0, 0, 0}, {F_DT, F_EH, 0, 0, 1}, {F_P, F_EEX, 0, 0, 0}, {F_EHT, F_CT, 0, 0, 1}},
    // C Hee^T - Hee^T C + P^H Heh^T - conj(Heh) P
    {{F_C, F_EE, 0, 0, 0}, {F_EET, F_CT, 0, 0, 1}, {F_PT, F_EH, 1, 0, 0}, {F_EH, F_PT, 1, 0, 1}},
    // D Hhh^T - Hhh^T D + conj(P) Heh - Heh^H P^T
    {{F_D, F_HH, 0, 0, 0}, {F_HHT, F_DT, 0, 0, 1}, {F_P, F_EHT, 1, 0, 0}, {F_EHT, F_P, 1, 0, 1}}};

// Into how many parts a product's K sequence (2 nkb K blocks) is cut, each a tile of its own whose
// partial result the finish adds.  Cost of p parts, in times of one K block: the waves of 152 CTAs
// (an SM each) times what a tile takes, its K blocks and 1.2 for its start and end; and for every
// part after the first the memory traffic and additions of its partial result, 0.15 for commutators
// and 2 for sources, whose reduction reads as much as the products write.  Measured: 1 x 512 (768
// tiles) 340 us uncut, 322 in two; 8 x 256 (1536 tiles) 326 uncut, 331 in two.
static int product_parts(long long units, int nkb, double part_cost = 0.15) {
  const int n = 2 * nkb;
  int best = 1;
  double least = 1e300;
  for (int p = 1; p <= std::min(n / 2, 8); ++p) {
    const double waves = (double)((units * p + 151) / 152);
    const double cost = waves * ((n + p - 1) / p + 1.2) + part_cost * (p - 1);
    if (cost < least) {
      least = cost;
      best = p;
    }
  }
  return best;
}

// forms planes of Nk x Nk matrices: slab of (form, plane, batch entry)
struct FormSet {
  __half* pl;
  int* e;
  int nk, nw;
  long long sl;
  __half* plane(int f) const { return pl + (long long)f * 2 * NS * nw * sl; }
  int* exps(int f) const { return e + (long long)f * nw * nk; }
};

static f64s::Job form_job(const FormSet& F, const TermDef& t, const int* alias) {
  f64s::Job j{};
  const int a = alias ? alias[t.a] : t.a, b = alias ? alias[t.b] : t.b;
  j.A = F.plane(a);
  j.B = F.plane(b);
  j.a_plane = j.b_plane = (long long)F.nw * F.sl;
  j.a_batch = j.b_batch = F.sl;
  j.a_pad = j.b_pad = pad_rows(F.nk);
  j.ea = F.exps(a);
  j.eb = F.exps(b);
  j.M = j.N = F.nk;
  j.nkb = k_blocks(F.nk);
  j.batch = F.nw;
  j.cplx = 1;
  j.conj_a = t.ca;
  j.conj_b = t.cb;
  j.neg = t.neg;
  j.ldo = F.nk;
  return j;
}

// the jobs of outputs [o0, o1) into part
static int form_products(const FormSet& F, int o0, int o1, const int* alias, int parts, double* part,
                         int* err, cudaStream_t s) {
  std::vector<f64s::Job> jobs;
  const long long cs = (long long)F.nw * F.nk * F.nk;
  for (int o = o0; o < o1; ++o)
    for (int t = 0; t < 4; ++t) {
      f64s::Job j = form_job(F, kTerms[o][t], alias);
      j.parts = parts;
      j.out = part + (((long long)(o - o0) * 4 + t) * parts) * 2 * cs;
      j.o_part = 2 * cs;
      j.o_comp = cs;
      j.o_batch = (long long)F.nk * F.nk;
      jobs.push_back(j);
    }
  return launch_f64_gemm(jobs.data(), (int)jobs.size(), err, s);
}

static int exchange(int nk, int nw, const double2* P, const double2* C, const double2* D,
                    const __half* tp, long long tp_plane, const int* et, long long et_n, __half* sp,
                    int* es, long long sl_m, long long sl_s, double* xsh, int* err,
                    cudaStream_t s) {
  const int nb = k_blocks(nk);
  int ny = 0;   // dd blocks of the band per t' block
  for (int i = 0; i < nb; ++i) {
    int cnt = 0;
    for (int j = shear_first(nk, 32 * i); 32 * j < 2 * nk; ++j)
      if (shear_live(nk, 32 * i, 32 * j)) cnt = j - shear_first(nk, 32 * i) + 1;
    ny = std::max(ny, cnt);
  }
  launch(k_f64_shear, dim3(nb, ny, 3 * nw), 256, 0, s, nk, nw, P, C, D, es, sp, sl_s);
  f64s::Job jobs[3];
  for (int n = 0; n < 3; ++n) {
    f64s::Job& j = jobs[n];
    j = f64s::Job{};
    j.A = tp + (long long)n * NS * tp_plane;
    j.a_plane = tp_plane;
    j.a_batch = sl_m;
    j.B = sp + (long long)n * NS * nw * sl_s;
    j.b_plane = (long long)nw * sl_s;
    j.b_batch = sl_s;
    j.a_pad = pad_rows(nk);
    j.b_pad = pad_rows(4 * nk);
    j.ea = et + n * et_n;
    j.eb = es + (long long)n * nw * (4 * nk - 2);
    j.M = nk;
    j.N = 4 * nk - 2;
    j.nkb = nb;
    j.batch = nw;
    j.parts = 1;
    j.band = nk;
    j.out = xsh + (long long)n * nw * 2 * nk * nk;
    j.o_batch = 2ll * nk * nk;
    j.ldo = 2 * nk;
  }
  return launch_f64_gemm(jobs, 3, err, s);
}

// ---------------------------------------------------------------------------
// context workspace

// Smallest Nk on the sliced products: below it the SIMT kernels take a few
// microseconds and the slices, padded to 128 x 64 tiles, do not pay.
constexpr int kMinNk = 32;
constexpr size_t kGroupBytes = 3ull << 30;   // pass workspace per bucket

// While another stream is being captured (in the default, global mode from any thread), this thread's
// allocations would fail and spoil that capture; in relaxed mode they do neither.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

bool f64_prepare(SbeCtx* c, cudaStream_t s) {
  if (c->f64) return true;
  if (c->f64_off) return false;
  for (const auto& W : c->wires)
    if (W.nk < kMinNk) return false;
  // no allocation inside a stream capture: such a first call takes the SIMT kernels
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
    cudaGetLastError();
    return false;
  }
  const RelaxedCapture relaxed;
  F64Work* w = new F64Work();
  c->f64 = w;
  bool ok = true;
  for (int i = 0; ok && i < c->nw;) {
    const WireDev& W0 = c->wires[c->order[i]];
    int j = i;
    while (j < c->nw && c->wires[c->order[j]].nk == W0.nk) ++j;
    F64Bucket m;
    const int nk = m.nk = W0.nk;
    m.nw = j - i;
    m.nr = W0.nr;
    m.bm = W0.off_mat;
    m.bv = W0.off_vec;
    m.br = W0.off_r;
    m.bkr = W0.off_kr;
    m.sl_m = f64s::slab(nk, nk);
    m.sl_s = f64s::slab(4 * nk, nk);
    m.sl_e = f64s::slab(m.nr, nk);
    const long long tm = (nk + 127) / 128, tiles = tm * ((nk + 63) / 64);
    const long long stiles = tm * ((m.nr + 63) / 64);
    m.group = 1;
    auto sizes = [&](int g, size_t* out) {
      const int parts = product_parts(24 * tiles * g, k_blocks(nk));
      const int sparts = product_parts(6 * stiles * g, k_blocks(nk), 2.0);
      out[0] = sizeof(__half) * F_N * 2 * NS * g * m.sl_m;                // forms
      out[1] = sizeof(__half) * 3 * NS * g * m.sl_s;                      // sheared
      // partial products, or the source products
      out[2] = sizeof(double) * std::max<size_t>(12ull * parts * 2 * g * nk * nk,
                                                 6ull * sparts * g * nk * m.nr);
      out[3] = sizeof(double) * 3 * g * 2 * nk * nk;                      // exchange
      out[4] = sizeof(int) * ((size_t)F_N * g * nk);
      out[5] = sizeof(int) * (size_t)3 * g * (4 * nk - 2);
      out[6] = sizeof(__half) * 3 * NS * m.nw * m.sl_m;                   // Toeplitz
      out[7] = sizeof(int) * (size_t)3 * m.nw * nk;
      out[8] = sizeof(__half) * 2 * NS * m.nw * m.sl_e;                   // E^T
      out[9] = sizeof(int) * (size_t)m.nw * m.nr;
      size_t t = 0;
      for (int k = 0; k < 10; ++k) t += (out[k] + 255) / 256 * 256;
      return t;
    };
    size_t sz[10];
    for (int g = m.nw; g > 1; g = (g + 1) / 2) {
      sizes(g, sz);
      size_t per = 0;
      for (int k = 0; k < 6; ++k) per += sz[k];
      if (per <= kGroupBytes) {
        m.group = g;
        break;
      }
    }
    const size_t total = sizes(m.group, sz);
    m.parts = product_parts(24 * tiles * m.group, k_blocks(nk));
    m.sparts = product_parts(6 * stiles * m.group, k_blocks(nk), 2.0);
    std::vector<WireDev> hw;
    for (int k = i; k < j; ++k) hw.push_back(c->wires[c->order[k]]);
    ok = cudaMalloc(&m.block, total) == cudaSuccess &&
         cudaMalloc(&m.dw, sizeof(WireDev) * m.nw) == cudaSuccess;
    if (ok) {
      char* p = static_cast<char*>(m.block);
      auto take = [&](int k) {
        char* r = p;
        p += (sz[k] + 255) / 256 * 256;
        return r;
      };
      m.pl = (__half*)take(0);
      m.sp = (__half*)take(1);
      m.part = (double*)take(2);
      m.xsh = (double*)take(3);
      m.ef = (int*)take(4);
      m.es = (int*)take(5);
      m.tp = (__half*)take(6);
      m.et = (int*)take(7);
      m.ep = (__half*)take(8);
      m.ee = (int*)take(9);
      // the sheared planes outside the band stay zero; rows past Nk of the other planes
      // only reach outputs that are not stored
      cudaMemsetAsync(m.block, 0, total, s);
      cudaMemcpyAsync(m.dw, hw.data(), sizeof(WireDev) * m.nw, cudaMemcpyHostToDevice, s);
      cudaStreamSynchronize(s);   // the host vector goes out of scope
      // E^T planes of the sources: Y[r][k] = Expikr[k][r]
      f64s::SliceArgs a{};
      a.f[0] = f64s::Form{c->expikr + m.bkr, nullptr, 1, 0, m.ep, m.ee};
      a.rows = m.nr;
      a.kdim = nk;
      a.ld = m.nr;
      a.batch = m.nw;
      a.src_batch = (long long)nk * m.nr;
      a.plane = (long long)m.nw * m.sl_e;
      a.dst_batch = m.sl_e;
      launch_f64_slice(a, 1, s);
    } else {
      cudaGetLastError();
    }
    w->b.push_back(m);
    i = j;
  }
  if (!ok) {
    // no room for the planes: the SIMT kernels need none
    f64_free(c);
    c->f64_off = 1;
    return false;
  }
  return true;
}

// Per-step operands: the Toeplitz planes of the screened interaction.
void f64_step_operands(SbeCtx* c, cudaStream_t s) {
  for (auto& m : work_of(c)->b)
    launch(k_f64_toeplitz, dim3((m.nk + 7) / 8, 3, m.nw), 256, 0, s, m.nk, m.nw, c->vs + 3 * m.bv,
           m.tp, m.et, m.sl_m);
}

static void state_forms(f64s::SliceArgs& a, const FormSet& F, const double2* P, const double2* C,
                        const double2* D) {
  const double2* x[3] = {P, C, D};
  for (int i = 0; i < 6; ++i)
    a.f[i] = f64s::Form{x[i / 2], nullptr, i & 1, peeled(i), F.plane(i), F.exps(i)};
}

static f64s::SliceArgs slice_args(const FormSet& F) {
  f64s::SliceArgs a{};
  a.rows = a.kdim = a.ld = F.nk;
  a.batch = F.nw;
  a.src_batch = (long long)F.nk * F.nk;
  a.plane = (long long)F.nw * F.sl;
  a.dst_batch = F.sl;
  a.add_f = kHbar;
  return a;
}

// One RHS evaluation of every wire at (P, C, D) with the wire-k field Ek; stage 0 stores
// dP, dC, dD, stages 1-4 apply the RK4 update (X: the step's state).
int f64_rhs(SbeCtx* c, const double2* P, const double2* C, const double2* D, const double2* Ek,
            int stage, double dt, double2* const* out, double2* const* X, cudaStream_t s) {
  bool exc = false;
  for (const auto& W : c->wires) exc = exc || (W.flags & SBE_F_EXCITONS);
  for (auto& m : work_of(c)->b)
    for (int w0 = 0; w0 < m.nw; w0 += m.group) {
      const int g = std::min(m.group, m.nw - w0), nk = m.nk;
      const long long mm = (long long)nk * nk, o = m.bm + w0 * mm, vo = m.bv + (long long)w0 * nk;
      const long long ro = m.br + (long long)w0 * m.nr;
      const FormSet F{m.pl, m.ef, nk, g, m.sl_m};
      launch(k_f64_diag, dim3((2 * nk - 1 + 3) / 4, 3, g), 128, 0, s, nk, P + o, C + o, D + o,
             c->tr + 4 * vo, m.es);
      int rc = SBE_OK;
      if (exc)
        rc = exchange(nk, g, P + o, C + o, D + o, m.tp + w0 * m.sl_m, (long long)m.nw * m.sl_m,
                      m.et + (long long)w0 * nk, (long long)m.nw * nk, m.sp, m.es, m.sl_m, m.sl_s,
                      m.xsh, c->f64_err, s);
      if (rc) return rc;
      HBuild h{};
      h.nk = nk;
      h.nr = m.nr;
      h.nw = g;
      h.wires = m.dw + w0;
      h.C = C + o;
      h.D = D + o;
      h.Ek = Ek ? Ek + 3 * ro : nullptr;
      h.vs = c->vs + 3 * vo;
      h.Ee = c->Ee + vo;
      h.Eh = c->Eh + vo;
      h.tr = c->tr + 4 * vo;
      h.xsh = reinterpret_cast<const double2*>(m.xsh);
      h.Heh = c->Heh + o;
      h.Hee = c->Hee + o;
      h.Hhh = c->Hhh + o;
      launch(k_f64_hbuild, dim3((nk + 127) / 128, nk, g), 128, 0, s, h);
      const double2* hm[3] = {c->Heh + o, c->Hee + o, c->Hhh + o};
      // the state's forms with the Hamiltonians' in one launch (two: 1 x 64 315 us a step, here
      // 289; 8 x 256 4.22 ms, 4.14)
      f64s::SliceArgs a = slice_args(F);
      state_forms(a, F, P + o, C + o, D + o);
      int nf = 6, alias[F_N];
      for (int i = 0; i < F_N; ++i) alias[i] = i;
      for (int i = 0; i < 6; ++i)
        a.f[nf++] = f64s::Form{hm[i / 2], nullptr, i & 1, peeled(F_EH + i), F.plane(F_EH + i),
                               F.exps(F_EH + i)};
      if (c->any_offdiag) {
        a.f[nf++] = f64s::Form{hm[1], c->dB + o, 0, 1, F.plane(F_EEX), F.exps(F_EEX)};
        a.f[nf++] = f64s::Form{hm[2], c->dA + o, 0, 1, F.plane(F_HHX), F.exps(F_HHX)};
      } else {
        alias[F_EEX] = F_EE;
        alias[F_HHX] = F_HH;
      }
      launch_f64_slice(a, nf, s);
      rc = form_products(F, 0, 3, alias, m.parts, m.part, c->f64_err, s);
      if (rc) return rc;
      Finish f{};
      f.nk = nk;
      f.nw = g;
      f.nsum = 4 * m.parts;
      f.stage = stage;
      f.dt = dt;
      f.dt6 = dt / 6.0;
      f.part = m.part;
      const double2* st[3] = {P + o, C + o, D + o};
      f.gamE = c->gamE + vo;
      f.gamH = c->gamH + vo;
      const long long n = c->tot_mat;
      for (int i = 0; i < 3; ++i) {
        f.X0[i] = st[i];
        f.H[i] = hm[i];
        f.out[i] = out ? out[i] + o : nullptr;
        f.X[i] = X ? X[i] + o : nullptr;
        f.acc[i] = c->kacc + i * n + o;
        f.xs[i] = c->xs + i * n + o;
      }
      launch(k_f64_finish, dim3((nk + 31) / 32, (nk + 7) / 8, 3 * g), dim3(32, 8), 0, s, f);
    }
  return cuda_check(cudaGetLastError(), "f64 rhs");
}

// ---------------------------------------------------------------------------
// sources

// Column sums of QWPolarization3 / QWRho5 (k_src_reduce) from the planar products
// G[n][part][re, im][wire][k][r], n = P E, C E, conj(D) E.  Block (16 r) x (32 k groups): thread
// (x, y) sums k = y, y + 32, ..., the partial sums are added in group order.
__global__ void __launch_bounds__(512) k_f64_src_reduce(const WireDev* wires, int nk, int nr, int nw,
                                                        int parts, const double2* E,
                                                        const double* G, const double* win,
                                                        double2* src) {
  pdl_enter();
  __shared__ double red[6][32][17];
  const int b = blockIdx.y, tx = threadIdx.x, ty = threadIdx.y, r = blockIdx.x * 16 + tx;
  const long long per = (long long)nk * nr, cs = (long long)nw * per;
  double s[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  if (r < nr) {
    const double2* e0 = E + (long long)b * per + r;
    const double* g0 = G + (long long)b * per + r;
#pragma unroll 4
    for (int k = ty; k < nk; k += 32) {
      const long long o = (long long)k * nr;
      const double2 e = e0[o];   // conj taken below
      double g[6];
#pragma unroll
      for (int i = 0; i < 6; ++i) {
        const double* q = g0 + ((long long)(i >> 1) * parts * 2 + (i & 1)) * cs + o;
        g[i] = q[0];
        for (int p = 1; p < parts; ++p) g[i] += q[2 * p * cs];
      }
      const double re = fma(e.x, g[0], e.y * g[1]);
      s[0] += (k & 1) ? -re : re;
      s[1] += re;
      s[2] = fma(e.x, g[2], fma(e.y, g[3], s[2]));
      s[3] = fma(e.x, g[3], fma(-e.y, g[2], s[3]));
      s[4] = fma(e.x, g[4], fma(e.y, g[5], s[4]));
      s[5] = fma(e.x, g[5], fma(-e.y, g[4], s[5]));
    }
  }
#pragma unroll
  for (int i = 0; i < 6; ++i) red[i][ty][tx] = s[i];
  __syncthreads();
  if (ty >= 6 || r >= nr) return;
  // row ty sums quantity ty
  double t = 0.0;
#pragma unroll
  for (int g = 0; g < 32; ++g) t += red[ty][g][tx];
  const WireDev& W = wires[b];
  const bool optics = (W.flags & SBE_F_OPTICS) != 0;
  const double w = win[(long long)b * nr + r], pf = 2 * W.ehint / W.area / W.L;
  double2* out = src + (long long)b * 5 * nr;
  double* od = reinterpret_cast<double*>(out);
  if (ty == 0) {
    out[r] = make_double2(optics ? W.dcv * t * w * pf : 0.0, 0.0);
  } else if (ty == 1) {
    out[nr + r] = make_double2(optics ? W.dcv * t * w * W.yw * pf : 0.0, 0.0);
    out[2 * nr + r] = make_double2(optics ? -W.dcv * t * w * W.zsign * pf : 0.0, 0.0);
  } else {
    od[2 * ((ty < 4 ? 3ll : 4ll) * nr + r) + (ty & 1)] = t * (w / (2.0 * W.L));
  }
}

int f64_sources(SbeCtx* c, const double2* P, const double2* C, const double2* D, double2* src,
                cudaStream_t s) {
  for (auto& m : work_of(c)->b)
    for (int w0 = 0; w0 < m.nw; w0 += m.group) {
      const int g = std::min(m.group, m.nw - w0), nk = m.nk, nr = m.nr;
      const long long mm = (long long)nk * nk, o = m.bm + w0 * mm, ro = m.br + (long long)w0 * nr;
      const long long ko = m.bkr + (long long)w0 * nk * nr;
      const FormSet F{m.pl, m.ef, nk, g, m.sl_m};
      const double2* x[3] = {P + o, C + o, D + o};
      f64s::SliceArgs a = slice_args(F);
      f64s::Job jobs[3];
      const long long cs = (long long)g * nk * nr;
      for (int i = 0; i < 3; ++i) {
        a.f[i] = f64s::Form{x[i], nullptr, 0, 0, F.plane(2 * i), F.exps(2 * i)};
        f64s::Job& j = jobs[i];
        j = f64s::Job{};
        j.A = F.plane(2 * i);
        j.a_plane = (long long)g * F.sl;
        j.a_batch = F.sl;
        j.B = m.ep + w0 * m.sl_e;
        j.b_plane = (long long)m.nw * m.sl_e;
        j.b_batch = m.sl_e;
        j.a_pad = pad_rows(nk);
        j.b_pad = pad_rows(nr);
        j.ea = F.exps(2 * i);
        j.eb = m.ee + (long long)w0 * nr;
        j.M = nk;
        j.N = nr;
        j.nkb = k_blocks(nk);
        j.batch = g;
        j.cplx = 1;
        j.conj_a = i == 2;
        j.parts = m.sparts;
        j.out = m.part + 2ll * i * m.sparts * cs;
        j.o_part = 2 * cs;
        j.o_comp = cs;
        j.o_batch = (long long)nk * nr;
        j.ldo = nr;
      }
      launch_f64_slice(a, 3, s);
      const int rc = launch_f64_gemm(jobs, 3, c->f64_err, s);
      if (rc) return rc;
      launch(k_f64_src_reduce, dim3((nr + 15) / 16, g), dim3(16, 32), 0, s, m.dw + w0, nk, nr, g,
             m.sparts, c->expikr + ko, m.part, c->window + ro, src + 5 * ro);
    }
  return cuda_check(cudaGetLastError(), "f64 sources");
}

// ---------------------------------------------------------------------------
// the single-wire functions

// Scratch of the calls without a context: a stream-ordered pool per device that keeps up
// to 64 MB between synchronisations (the planes of Nk = 400 take 58 MB) and gives the rest
// back.  Allocations and releases are ordered on the caller's stream, so calls of any
// threads and streams may overlap.
static cudaMemPool_t scratch_pool() {
  static std::mutex mu;
  static std::map<int, cudaMemPool_t> pools;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
  std::lock_guard<std::mutex> lock(mu);
  auto it = pools.find(dev);
  if (it != pools.end()) return it->second;
  const RelaxedCapture relaxed;
  cudaMemPoolProps pr{};
  pr.allocType = cudaMemAllocationTypePinned;
  pr.location.type = cudaMemLocationTypeDevice;
  pr.location.id = dev;
  cudaMemPool_t p = nullptr;
  if (cudaMemPoolCreate(&p, &pr) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  unsigned long long keep = 64ull << 20;
  cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);
  pools[dev] = p;
  return p;
}

// One block of stream-ordered scratch (a word of it takes the products' error flag: the calls have
// no context that could report it, their outputs are NaN then); null when there is no room or the stream is being
// captured (the callers then take the SIMT kernels).
struct Scratch {
  char* p = nullptr;
  size_t off = 0;
  cudaStream_t s;
  Scratch(size_t bytes, cudaStream_t s_) : s(s_) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    cudaMemPool_t pool = nullptr;
    if (cudaStreamIsCapturing(s, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone ||
        !(pool = scratch_pool()) ||
        cudaMallocFromPoolAsync((void**)&p, bytes, pool, s) != cudaSuccess) {
      cudaGetLastError();
      p = nullptr;
    }
  }
  ~Scratch() {
    if (p) cudaFreeAsync(p, s);
  }
  template <typename T>
  T* take(size_t n) {
    T* r = reinterpret_cast<T*>(p + off);
    off += (sizeof(T) * n + 255) / 256 * 256;
    return r;
  }
};

bool f64_rhs_single(int which, int nk, const double2* C, const double2* D, const double2* P,
                    const double2* Heh, const double2* Hee, const double2* Hhh, const double* gamE,
                    const double* gamH, const double2* offp, double2* out, cudaStream_t s, int* rc) {
  if (nk < kMinNk) return false;
  const long long tiles = (long long)((nk + 127) / 128) * ((nk + 63) / 64), mm = (long long)nk * nk;
  const int parts = product_parts(8 * tiles, k_blocks(nk));
  // the forms this output's terms use, in their own slots
  const double2* mats[6] = {P, C, D, Heh, Hee, Hhh};
  int alias[F_N], slot[F_N], nf = 0;
  for (int i = 0; i < F_N; ++i) slot[i] = -1;
  f64s::SliceArgs a{};
  for (int t = 0; t < 4; ++t)
    for (int f : {kTerms[which][t].a, kTerms[which][t].b}) {
      const int g = f == F_EEX ? F_EE : f == F_HHX ? F_HH : f;
      if (slot[g] < 0) {
        slot[g] = nf;
        a.f[nf].src = mats[g / 2];
        a.f[nf].transpose = g & 1;
        a.f[nf].peel = peeled(g);
        ++nf;
      }
      alias[f] = slot[g];
    }
  const long long sl = f64s::slab(nk, nk);
  Scratch w(sizeof(__half) * nf * 2 * NS * sl + sizeof(int) * nf * nk +
                sizeof(double) * 8 * parts * mm + 1024, s);
  if (!w.p) return false;
  const FormSet F{w.take<__half>((size_t)nf * 2 * NS * sl), w.take<int>((size_t)nf * nk), nk, 1, sl};
  double* part = w.take<double>((size_t)8 * parts * mm);
  for (int i = 0; i < nf; ++i) {
    a.f[i].dst = F.plane(i);
    a.f[i].e = F.exps(i);
  }
  a.rows = a.kdim = a.ld = nk;
  a.batch = 1;
  a.src_batch = mm;
  a.plane = a.dst_batch = sl;
  launch_f64_slice(a, nf, s);
  *rc = form_products(F, which, which + 1, alias, parts, part, w.take<int>(1), s);
  if (*rc) return true;
  Finish f{};
  f.nk = nk;
  f.nw = 1;
  f.nsum = 4 * parts;
  f.first = which;
  f.part = part;
  for (int i = 0; i < 3; ++i) {
    f.X0[i] = mats[i];
    f.H[i] = mats[3 + i];
  }
  f.offp = offp;
  f.gamE = gamE;
  f.gamH = gamH;
  f.out[which] = out;
  launch(k_f64_finish, dim3((nk + 31) / 32, (nk + 7) / 8, 1), dim3(32, 8), 0, s, f);
  *rc = cuda_check(cudaGetLastError(), "f64 rhs single");
  return true;
}

bool f64_calch_single(int nk, const double2* Meh, const double2* Wee, const double2* Whh,
                      const double2* C, const double2* D, const double2* P, const double* VC,
                      const double* Ee, const double* Eh, double gap, int excitons, int lf,
                      int freepot, double2* Heh, double2* Hee, double2* Hhh, cudaStream_t s, int* rc) {
  if (nk < kMinNk || !excitons) return false;
  const long long sl = f64s::slab(nk, nk), ss = f64s::slab(4 * nk, nk), mm = (long long)nk * nk;
  Scratch w(sizeof(__half) * 3 * NS * (sl + ss) + sizeof(int) * 3 * (5 * nk) +
                sizeof(double) * (6 * mm + 3 * nk) + sizeof(double2) * 4 * nk + 4096, s);
  if (!w.p) return false;
  __half *tp = w.take<__half>(3 * NS * sl), *sp = w.take<__half>(3 * NS * ss);
  int *et = w.take<int>(3 * nk), *es = w.take<int>(3 * (4 * nk - 2));
  double *xsh = w.take<double>(6 * mm), *vq = w.take<double>(3 * nk);
  double2* tr = w.take<double2>(4 * nk);
  launch_vq_from_vc(nk, VC, vq, s);
  // blocks of the sheared planes outside the band are not written by the pass
  cudaMemsetAsync(sp, 0, sizeof(__half) * 3 * NS * ss, s);
  launch(k_f64_diag, dim3((2 * nk - 1 + 3) / 4, 3, 1), 128, 0, s, nk, P, C, D, tr, es);
  launch(k_f64_toeplitz, dim3((nk + 7) / 8, 3, 1), 256, 0, s, nk, 1, vq, tp, et, sl);
  *rc = exchange(nk, 1, P, C, D, tp, sl, et, nk, sp, es, sl, ss, xsh, w.take<int>(1), s);
  if (*rc) return true;
  HBuild h{};
  h.nk = nk;
  h.nr = 2 * nk + 2;
  h.nw = 1;
  h.C = C;
  h.D = D;
  h.vs = vq;
  h.Ee = Ee;
  h.Eh = Eh;
  h.tr = tr;
  h.xsh = reinterpret_cast<const double2*>(xsh);
  h.Meh = Meh;
  h.Wee = Wee;
  h.Whh = Whh;
  h.gap = gap;
  h.excitons = excitons;
  h.lf = lf;
  h.freepot = freepot;
  h.Heh = Heh;
  h.Hee = Hee;
  h.Hhh = Hhh;
  launch(k_f64_hbuild, dim3((nk + 127) / 128, nk, 1), 128, 0, s, h);
  *rc = cuda_check(cudaGetLastError(), "sbe_calch");
  return true;
}

}  // namespace sbe
