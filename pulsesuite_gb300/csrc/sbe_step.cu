// Time stepping of every wire: the reference leapfrog update, relaxation and
// charge normalisation, RK4 stage updates, the polarisation / charge sources and
// the field resampling between the propagation grid and the wire grid (FP64).
#include "cluster_sum.cuh"
#include "fp_bits.cuh"
#include "sbe_ctx.cuh"
#include "spline.cuh"

namespace sbe {

// ---------------------------------------------------------------------------
// SBEs.py:5673-5675: X3 = X1 + 2 dt dX for P, C, D; X3 is written into the
// level-1 buffers (their old contents are not needed any more).
__global__ void k_leap_update(const WireDev* wires, double2* L1p, const double2* L2p,
                              const double2* dP, double2* L1c, const double2* L2c,
                              const double2* dC, double2* L1d, const double2* L2d,
                              const double2* dD, double dt) {
  pdl_enter();
  const WireDev W = wires[blockIdx.y];
  long long n = (long long)W.nk * W.nk;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    long long o = W.off_mat + i;
    double2 a = L2p[o], d = dP[o];
    L1p[o] = make_double2(a.x + d.x * dt * 2.0, a.y + d.y * dt * 2.0);
    a = L2c[o]; d = dC[o];
    L1c[o] = make_double2(a.x + d.x * dt * 2.0, a.y + d.y * dt * 2.0);
    a = L2d[o]; d = dD[o];
    L1d[o] = make_double2(a.x + d.x * dt * 2.0, a.y + d.y * dt * 2.0);
  }
}

// SBEs.py:5704-5706 and _checkin (5070-5080): with X3 held in level 1,
// new level1 = old level2, level2 = (old level2 + X3)/2, level3 = X3.
__global__ void k_leap_shuffle(const WireDev* wires, double2* L1, double2* L2, double2* L3) {
  pdl_enter();
  const WireDev W = wires[blockIdx.y];
  long long n = (long long)W.nk * W.nk;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    long long o = W.off_mat + i;
    double2 a = L2[o], b = L1[o];
    L1[o] = a;
    L2[o] = make_double2((a.x + b.x) / 2.0, (a.y + b.y) / 2.0);
    L3[o] = b;
  }
}

// phonons.py:140-268 MBPE / MBPH for row k of every wire, with the couplings of the
// preparation: Vep = VC[:,:,1]/E1D*Vscale (VC already divided by E1D once: the quirk is
// kept).  ne, nh: Re of the vectors, or (diag) of the diagonals of the matrices C3, D3.
__global__ void __launch_bounds__(128) k_phonon_rates(const WireDev* wires, int w_only,
                                                      const double2* nev, const double2* nhv,
                                                      int diag, const double* vph, const double* EP,
                                                      const double* HP, double* wrate) {
  pdl_enter();
  const WireDev& W = wires[w_only >= 0 ? w_only : blockIdx.y];
  const int nk = W.nk;
  int k = blockIdx.x;
  if (k >= nk) return;
  if (!(W.flags & SBE_F_PHONON)) {
    // no phonon rates: the carrier-carrier rates (EHs) are added to zeros
    if (threadIdx.x < 4) wrate[4 * W.off_vec + threadIdx.x * nk + k] = 0.0;
    return;
  }
  const double* ve = vph + 2 * W.off_vec;
  const double* vh = ve + nk;
  const double2* pe = nev + (diag ? W.off_mat : W.off_vec);
  const double2* ph = nhv + (diag ? W.off_mat : W.off_vec);
  const long long st = diag ? nk + 1 : 1;
  const double* EPw = EP + W.off_mat;
  const double* HPw = HP + W.off_mat;
  double r[4] = {0.0, 0.0, 0.0, 0.0};
  for (int i = threadIdx.x; i < nk; i += blockDim.x) {
    if (i <= k) {   // electrons: Vep[k, i] (nonzero for k >= i)
      const double n = pe[i * st].x, v = ve[k - i];
      r[0] += v * n * EPw[(long long)k * nk + i];
      r[1] += v * (1.0 - n) * EPw[(long long)i * nk + k];
    }
    if (i >= k) {   // holes: Vhp[i, k] (nonzero for i >= k)
      const double n = ph[i * st].x, v = vh[i - k];
      r[2] += v * n * HPw[(long long)k * nk + i];
      r[3] += v * (1.0 - n) * HPw[(long long)i * nk + k];
    }
  }
  __shared__ double red[4][4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    for (int o = 16; o > 0; o >>= 1) r[j] += __shfl_down_sync(0xffffffffu, r[j], o);
    if ((threadIdx.x & 31) == 0) red[j][threadIdx.x >> 5] = r[j];
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    const double* q = red[threadIdx.x];
    wrate[4 * W.off_vec + threadIdx.x * nk + k] = (q[0] + q[1]) + (q[2] + q[3]);
  }
}

// SBEs.py:5677-5702 + 5276-5325: relaxation of the diagonals with the phonon
// in/out rates, then the charge normalisation ne = |C_kk| scaled to the common
// mean.  One block per wire.  The normalised occupations are left in ne/nh for
// the sources.
__device__ __forceinline__ double2 cexp_d(double2 z) {
  const double m = exp(z.x);
  double sn, cs;
  sincos(z.y, &sn, &cs);
  return make_double2(m * cs, m * sn);
}

// mode 0: relaxation and normalisation; 1: relaxation only (the relaxed complex
// diagonals back into C3, D3); 2: normalisation only.  One cluster per wire: the four
// exponentials and divisions per k are bound by the FP64 pipes of its SMs, a warp's
// instruction by its 64 clocks, so they run side by side in a warp's lanes (1 x 64: 12.6 -> 6.7 us).
__global__ void __cluster_dims__(kCluster, 1, 1) __launch_bounds__(256)
    k_relax_norm(const WireDev* wires, double2* C3, double2* D3, const double* wrate,
                 const double* rsp, double dt, double2* ne_out, double2* nh_out, double* charge,
                 int mode) {
  pdl_enter();
  const WireDev& W = wires[blockIdx.y];
  // four lanes per k: electrons and holes, the two exponentials and then the two components
  const int nk = W.nk, sub = threadIdx.x & 3, kst = kCluster * 64;
  const int k0 = blockIdx.x + kCluster * (threadIdx.x >> 2);
  const unsigned quad = 0xFu << (threadIdx.x & 28);
  const bool hole = sub >= 2, im = sub & 1;
  double2* X3 = hole ? D3 : C3;
  double2* x_out = hole ? nh_out : ne_out;
  const bool relax = mode != 2 && (W.flags & (SBE_F_PHONON | SBE_F_EHS)) != 0;
  // the decay is part of the relaxation, which runs only with Phonon or EHs
  // (SBEs.py:5677, 5322)
  const bool recomb = relax && (W.flags & SBE_F_RECOMB) != 0;
  double sum = 0.0;
  for (int k = k0; k < nk; k += kst) {
    const long long o = W.off_mat + (long long)k * nk + k;
    double2 n = X3[o];
    if (relax) {
      const double* wr = wrate + 4 * W.off_vec + (hole ? 2 * nk : 0);
      const double wi = wr[k], wo = wr[nk + k], w = wi + wo;
      const double mine = exp(im ? w * dt : -w * dt);
      const double other = __shfl_xor_sync(quad, mine, 1);
      const double em = im ? other : mine, ep = im ? mine : other;
      const double first = im ? n.y : -1 + ep + n.x, x = im ? n.y : n.x;
      const double y = em * (first * wi + x * wo) / (w + kSmall);
      const double z = __shfl_xor_sync(quad, y, 1);
      n = im ? make_double2(z, y) : make_double2(y, z);
    }
    if (recomb) {
      // SBEs.py:5322-5325: ne exp(-Rsp nh dt), then nh exp(-Rsp ne dt) with the new ne
      // (complex occupations, complex exponential)
      const double r = rsp[W.off_vec + k];
      for (int turn = 0; turn < 2; ++turn) {
        const double2 u = make_double2(__shfl_xor_sync(quad, n.x, 2), __shfl_xor_sync(quad, n.y, 2));
        if (hole == (turn == 1)) n = cmul(n, cexp_d(make_double2(-r * u.x * dt, -r * u.y * dt)));
      }
    }
    if (mode == 1) {
      __syncwarp(quad);
      if (!im) X3[o] = n;
      continue;
    }
    const double a = cabs_d(n);
    if (!im) {
      x_out[W.off_vec + k] = make_double2(a, 0.0);
      sum += a;
    }
  }
  if (mode == 1) return;   // uniform over the cluster
  double se = hole ? 0.0 : sum, sh = hole ? sum : 0.0;
  cluster_sum2(se, sh, blockIdx.x + kCluster * ((threadIdx.x & ~31) >> 2) < nk);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    // the carrier numbers before the normalisation: their difference is what this
    // step's relaxation and rounding left of the electron-hole balance
    charge[2 * blockIdx.y] = se;
    charge[2 * blockIdx.y + 1] = sh;
  }
  if (im || k0 >= nk) return;
  const double f = (se + sh) / 2.0 / ((hole ? sh : se) + kSmall);
  for (int k = k0; k < nk; k += kst) {
    const double2 a = make_double2(x_out[W.off_vec + k].x * f, 0.0);
    x_out[W.off_vec + k] = a;
    X3[W.off_mat + (long long)k * nk + k] = a;
  }
}

bool any_ehs(const SbeCtx* c) {
  for (const auto& W : c->wires)
    if (W.flags & SBE_F_EHS) return true;
  return false;
}

void launch_relax_norm(SbeCtx* c, double2* P3, double2* C3, double2* D3, const double2* Ek,
                       double dt, cudaStream_t s) {
  if (any_ehs(c)) launch_extract_diag(c, C3, D3, s);   // for the carrier-carrier rates
  launch(k_phonon_rates, dim3(c->nk_max, c->nw), 128, 0, s, c->d_wires, -1, C3, D3, 1, c->vph,
         c->EP, c->HP, c->wrate);
  launch_mbc_rates(c, -1, s);
  launch_relax_only(c, P3, C3, D3, Ek, dt, s);
}

// relaxation (rates already in c->wrate), DC transport and normalisation
// (SBEs.py:5677-5702: relaxation, Transport of C3, D3, p3, charge normalisation)
void launch_relax_only(SbeCtx* c, double2* P3, double2* C3, double2* D3, const double2* Ek,
                       double dt, cudaStream_t s) {
  if (!any_dc(c)) {
    launch(k_relax_norm, dim3(kCluster, c->nw), 256, 0, s, c->d_wires, C3, D3, c->wrate, c->rsp, dt,
           c->ne, c->nh, c->charge, 0);
    return;
  }
  launch(k_relax_norm, dim3(kCluster, c->nw), 256, 0, s, c->d_wires, C3, D3, c->wrate, c->rsp, dt,
         c->ne, c->nh, c->charge, 1);
  launch_dc_transport(c, P3, C3, D3, Ek, dt, s);
  launch(k_relax_norm, dim3(kCluster, c->nw), 256, 0, s, c->d_wires, C3, D3, c->wrate, c->rsp, dt,
         c->ne, c->nh, c->charge, 2);
}

void launch_phonon_rates_one(SbeCtx* c, int w, cudaStream_t s) {
  launch(k_phonon_rates, dim3(c->wires[w].nk, 1), 128, 0, s, c->d_wires, w, c->ne, c->nh, 0, c->vph,
         c->EP, c->HP, c->wrate);
}

void launch_leapfrog(SbeCtx* c, double2* const* st, const double2* Ek, double dt,
                     cudaStream_t s) {
  // st: YY1, YY2, YY3, CC1, CC2, CC3, DD1, DD2, DD3
  int blocks = (int)std::min<long long>(((long long)c->nk_max * c->nk_max + 255) / 256, 4096);
  dim3 g(blocks, c->nw);
  launch(k_leap_update, g, 256, 0, s, c->d_wires, st[0], st[1], c->dP, st[3], st[4], c->dC, st[6],
         st[7], c->dD, dt);
  launch_relax_norm(c, st[0], st[3], st[6], Ek, dt, s);
}

void launch_leap_shuffle(SbeCtx* c, double2* const* st, cudaStream_t s) {
  int blocks = (int)std::min<long long>(((long long)c->nk_max * c->nk_max + 255) / 256, 4096);
  dim3 g(blocks, c->nw);
  launch(k_leap_shuffle, g, 256, 0, s, c->d_wires, st[0], st[1], st[2]);
  launch(k_leap_shuffle, g, 256, 0, s, c->d_wires, st[3], st[4], st[5]);
  launch(k_leap_shuffle, g, 256, 0, s, c->d_wires, st[6], st[7], st[8]);
}

// ---------------------------------------------------------------------------
// Sources.  qwoptics.py:50-76 (QWPolarization3) with Xvc0[kh,ke] = dcv (-1)^kh,
// Yvc0 = dcv, Zvc0 = -dcv (qwoptics.py:618-626) reduces to G = p E (E = Expikr)
// and column sums over kh; qwoptics.py:361-374 (QWRho5) to C E and conj(D) E.
// Output per wire: 5 x Nr c128 [Px, Py, Pz, re, rh] in real space (the
// reference's FFTG here is undone by the iFFTG of QW2Prop).
__global__ void k_src_reduce(const WireDev* wires, int w_only, const double2* expikr,
                             const double2* G, long long tot_kr, const double* win, double2* src) {
  pdl_enter();
  const WireDev W = wires[w_only >= 0 ? w_only : blockIdx.y];
  int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= W.nr) return;
  const int nk = W.nk, nr = W.nr;
  const double2* E = expikr + W.off_kr;
  const double2* Gp = G + W.off_kr;
  const double2* Gc = G + tot_kr + W.off_kr;
  const double2* Gd = G + 2 * tot_kr + W.off_kr;
  double sx = 0.0, sy = 0.0;
  double2 se = make_double2(0, 0), sh = make_double2(0, 0);
  for (int k = 0; k < nk; ++k) {
    double2 e = cconj(E[(long long)k * nr + r]);
    double2 gp = Gp[(long long)k * nr + r];
    double re_part = e.x * gp.x - e.y * gp.y;
    sx += (k & 1) ? -re_part : re_part;
    sy += re_part;
    se = cadd(se, cmul(e, Gc[(long long)k * nr + r]));
    sh = cadd(sh, cmul(e, Gd[(long long)k * nr + r]));
  }
  double w = win[W.off_r + r];
  double2* out = src + 5 * W.off_r;
  bool optics = (W.flags & SBE_F_OPTICS) != 0;
  double px = optics ? (W.dcv * sx) * w : 0.0;
  double py = optics ? (W.dcv * sy) * w * W.yw : 0.0;
  double pz = optics ? (-W.dcv * sy) * w * W.zsign : 0.0;
  out[r] = make_double2(px * 2 * W.ehint / W.area / W.L, 0.0);
  out[nr + r] = make_double2(py * 2 * W.ehint / W.area / W.L, 0.0);
  out[2 * nr + r] = make_double2(pz * 2 * W.ehint / W.area / W.L, 0.0);
  out[3 * nr + r] = cscale(se, w / (2.0 * W.L));
  out[4 * nr + r] = cscale(sh, w / (2.0 * W.L));
}

// qwoptics.py:1062-1068 boundary-mean subtraction and renormalisation, then
// SBEs.py:5749-5750 (x 2 e0 ehint / area).  One cluster per wire (FP64 square roots); every
// block forms the carrier sums and boundary means itself, the first cluster barrier keeps
// the boundary values from being overwritten before all have read them.
__global__ void __cluster_dims__(kCluster, 1, 1) __launch_bounds__(256)
    k_src_final(const WireDev* wires, int w_only, const double* r, const double2* ne,
                const double2* nh, double2* src) {
  pdl_enter();
  const WireDev& W = wires[w_only >= 0 ? w_only : blockIdx.y];
  // two lanes per point: electron and hole density
  const int nr = W.nr, nk = W.nk, st = kCluster * 128;
  const int j0 = blockIdx.x + kCluster * (threadIdx.x >> 1);
  const bool hole = threadIdx.x & 1;
  double2* re = src + 5 * W.off_r + 3 * nr;
  double2* rh = re + nr;
  double2* rho = hole ? rh : re;
  if (!(W.flags & SBE_F_LF)) {
    for (int j = j0; j < nr; j += st) rho[j] = make_double2(0, 0);
    return;
  }
  double v[4] = {0, 0, 0, 0};   // carrier sums, boundary sums
  for (int k = threadIdx.x; k < nk; k += 256) {
    v[0] += cabs_d(ne[W.off_vec + k]);
    v[1] += cabs_d(nh[W.off_vec + k]);
  }
  // sum(re[0:10]) + sum(re[Nr-10:Nr]): an index in both slices counts twice
  if (threadIdx.x < 20) {
    const int j = threadIdx.x < 10 ? threadIdx.x : nr - 20 + threadIdx.x;
    v[2] = re[j].x;
    v[3] = rh[j].x;
  }
  block_sums(v, (threadIdx.x & ~31) < nk || threadIdx.x < 32);
  const bool live = blockIdx.x + kCluster * ((threadIdx.x & ~31) >> 1) < nr;
  double sum = 0.0, bnd = 0.0;
  if (live) {
    bnd = div_by(hole ? v[3] : v[2], 20.0, 0.05);
    for (int j = j0; j < nr; j += st) {
      const double2 x = rho[j];
      sum += cabs_d(make_double2(x.x - bnd, x.y));
    }
  }
  double ae = hole ? 0.0 : sum, ah = hole ? sum : 0.0;
  cluster_sum2(ae, ah, live);
  if (j0 >= nr) return;
  const double* rw = r + W.off_r;
  const double dr = rw[1] - rw[0], N = (hole ? v[1] : v[0]) + 1e-50;
  const double f = W.rho_scale * (N / ((hole ? ah : ae) * dr + kQwSmall));
  for (int j = j0; j < nr; j += st) {
    const double2 x = rho[j];
    rho[j] = make_double2((x.x - bnd) * f, x.y * f);
  }
}

void launch_sources(SbeCtx* c, const double2* P, const double2* C, const double2* D,
                    const double2* ne, const double2* nh, double2* src, cudaStream_t s,
                    int w_only) {
  const double2 one = make_double2(1.0, 0.0);
  const double2* mats[3] = {P, C, D};
  for (int i = 0; i < 3; ++i) {
    GemmBatch b{};
    b.w_only = w_only;
    b.nterms = 1;
    b.t[0].A = mats[i];
    b.t[0].B = nullptr;
    b.t[0].opA = (i == 2) ? OP_C : OP_N;
    b.t[0].opB = OP_N;
    b.t[0].realA = 0;
    b.t[0].alpha = one;
    b.out = c->G + i * c->tot_kr;
    b.epi = 0;
    launch_sources_gemm64(c, b, s);
  }
  int nb = w_only >= 0 ? 1 : c->nw;
  (void)nb;
  launch(k_src_reduce, dim3((c->nr_max + 127) / 128, nb), 128, 0, s, c->d_wires, w_only, c->expikr,
         c->G, c->tot_kr, c->window, src);
  launch(k_src_final, dim3(kCluster, nb), 256, 0, s, c->d_wires, w_only, c->r, ne, nh, src);
}

// ---------------------------------------------------------------------------
// RK4 (classical tableau) over the packed state, FP64.  stage s in 1..4 uses the
// RHS in c->dP/dC/dD:  s=1: acc = k;   xs = X + dt/2 k
//                      s=2: acc += 2k; xs = X + dt/2 k
//                      s=3: acc += 2k; xs = X + dt k
//                      s=4: X += dt/6 (acc + k)
__global__ void k_rk4_axpy(long long n, int stage, double dt, double2* X, double2* acc,
                           double2* xs, const double2* k) {
  pdl_enter();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    double2 kv = k[i];
    if (stage == 1) {
      acc[i] = kv;
      double2 x = X[i];
      xs[i] = make_double2(x.x + 0.5 * dt * kv.x, x.y + 0.5 * dt * kv.y);
    } else if (stage == 2 || stage == 3) {
      double2 a = acc[i];
      acc[i] = make_double2(a.x + 2.0 * kv.x, a.y + 2.0 * kv.y);
      double f = stage == 2 ? 0.5 * dt : dt;
      double2 x = X[i];
      xs[i] = make_double2(x.x + f * kv.x, x.y + f * kv.y);
    } else {
      double2 a = acc[i], x = X[i];
      X[i] = make_double2(x.x + dt / 6.0 * (a.x + kv.x), x.y + dt / 6.0 * (a.y + kv.y));
    }
  }
}

void launch_rk4_axpy(SbeCtx* c, int stage, double dt, double2* P, double2* C, double2* D,
                     cudaStream_t s) {
  long long n = c->tot_mat;
  int blocks = (int)std::min<long long>((n + 255) / 256, 8192);
  double2* X[3] = {P, C, D};
  double2* K[3] = {c->dP, c->dC, c->dD};
  for (int i = 0; i < 3; ++i)
    launch(k_rk4_axpy, blocks, 256, 0, s, n, stage, dt, X[i], c->kacc + i * n, c->xs + i * n, K[i]);
}

__global__ void k_stage_field(long long n, const double2* Ek0, const double2* dEk, double frac,
                              double2* out) {
  pdl_enter();
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  double2 a = Ek0[i];
  if (dEk) {
    double2 b = dEk[i];
    a.x += frac * b.x;
    a.y += frac * b.y;
  }
  out[i] = a;
}

void launch_stage_field(SbeCtx* c, const double2* Ek0, const double2* dEk, double frac,
                        cudaStream_t s) {
  long long n = 3 * c->tot_r;
  launch(k_stage_field, (int)((n + 255) / 256), 256, 0, s, n, Ek0, dEk, frac, c->ekst);
}

// ---------------------------------------------------------------------------
// Cubic spline resampling, spliner.py:153-189 rescale_1D_dpc with the
// Forsythe-Malcolm-Moler coefficients of spline_dpc (spliner.py:1329-1394, spline.cu) and
// the binary search of locate (spliner.py:1137-1167).  Two or three knots have their own
// formulas: one thread per field.
__device__ void fmm_spline(int n, const double* x, const double2* y, double2* b, double2* c,
                           double2* d) {
  if (n < 3) {
    double2 s = cscale(csub(y[1], y[0]), 1.0 / (x[1] - x[0]));
    b[0] = s; b[1] = s;
    c[0] = c[1] = d[0] = d[1] = make_double2(0, 0);
    return;
  }
  d[0] = make_double2(x[1] - x[0], 0);
  c[1] = cscale(csub(y[1], y[0]), 1.0 / d[0].x);
  for (int i = 1; i < n - 1; ++i) {
    d[i] = make_double2(x[i + 1] - x[i], 0);
    b[i] = make_double2(2.0 * (d[i - 1].x + d[i].x), 0);
    double2 t = csub(y[i + 1], y[i]);
    c[i + 1] = make_double2(t.x / d[i].x, t.y / d[i].x);
    c[i] = csub(c[i + 1], c[i]);
  }
  b[0] = make_double2(-d[0].x, 0);
  b[n - 1] = make_double2(-d[n - 2].x, 0);
  c[0] = make_double2(0, 0);
  c[n - 1] = make_double2(0, 0);
  if (n != 3) {
    double2 c0 = csub(cscale(c[2], 1.0 / (x[3] - x[1])), cscale(c[1], 1.0 / (x[2] - x[0])));
    double2 cn = csub(cscale(c[n - 2], 1.0 / (x[n - 1] - x[n - 3])),
                      cscale(c[n - 3], 1.0 / (x[n - 2] - x[n - 4])));
    c[0] = cscale(c0, d[0].x * d[0].x / (x[3] - x[0]));
    c[n - 1] = cscale(cn, -d[n - 2].x * d[n - 2].x / (x[n - 1] - x[n - 4]));
  }
  for (int i = 1; i < n; ++i) {
    double t = d[i - 1].x / b[i - 1].x;
    b[i].x = b[i].x - t * d[i - 1].x;
    c[i] = csub(c[i], cscale(c[i - 1], t));
  }
  c[n - 1] = cscale(c[n - 1], 1.0 / b[n - 1].x);
  for (int i = n - 2; i >= 0; --i) {
    double2 t = csub(c[i], cscale(c[i + 1], d[i].x));
    c[i] = make_double2(t.x / b[i].x, t.y / b[i].x);
  }
  {
    double2 t = csub(y[n - 1], y[n - 2]);
    double2 u = cadd(c[n - 2], cscale(c[n - 1], 2.0));
    b[n - 1] = cadd(make_double2(t.x / d[n - 2].x, t.y / d[n - 2].x), cscale(u, d[n - 2].x));
  }
  for (int i = 0; i < n - 1; ++i) {
    double di = d[i].x;
    double2 t = csub(y[i + 1], y[i]);
    double2 u = cadd(c[i + 1], cscale(c[i], 2.0));
    b[i] = csub(make_double2(t.x / di, t.y / di), cscale(u, di));
    double2 v = csub(c[i + 1], c[i]);
    d[i] = make_double2(v.x / di, v.y / di);
    c[i] = cscale(c[i], 3.0);
  }
  c[n - 1] = cscale(c[n - 1], 3.0);
  d[n - 1] = d[n - 2];
}

__global__ void k_spline_coef(int n, const double* x, const double2* y, int nf, double2* coef) {
  pdl_enter();
  int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= nf) return;
  double2* b = coef + (long long)f * 3 * n;
  fmm_spline(n, x, y + (long long)f * n, b, b + n, b + 2 * n);
}

static void spline_coefs(int n, const double* x, const double2* y, int nf, double2* coef, int* bad,
                         cudaStream_t s) {
  if (n < kSplMin) {
    launch(k_spline_coef, 1, 32, 0, s, n, x, y, nf, coef);
    return;
  }
  SplBatch b{};
  b.X = x;
  b.Y = y;
  b.coef = coef;
  b.n0 = n;
  b.nf = nf;
  b.bad = bad;
  launch_splines(b, 1, n, s);
}

// evaluate nf splines (knots x0, n0) at x1 (n1 points); values outside
// [min x0, max x0] are 0; optional window multiply and real part.  The block finds the
// knots' range together.  A part of a field (real, imaginary) with a coefficient that is not finite
// is NaN everywhere, as a solve from end to end leaves it.
__global__ void __launch_bounds__(128) k_spline_eval(int n0, const double* x0, const double2* y0,
                                                     const double2* coef, const int* bad, int n1,
                                                     const double* x1, int nf, const double* win,
                                                     int real_part, double2* out) {
  pdl_enter();
  __shared__ double rlo[4], rhi[4];
  __shared__ int rbad[4];
  double lo = x0[0], hi = lo;
  for (int i = threadIdx.x; i < n0; i += 128) {
    const double x = x0[i];
    lo = fmin(lo, x);
    hi = fmax(hi, x);
  }
  int nan = 0;
  if (n0 >= kSplMin)
    for (int i = threadIdx.x; i < spl_tiles(n0); i += 128) nan |= bad[i];
  nan = __reduce_or_sync(0xffffffffu, nan);
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if ((threadIdx.x & 31) == 0) {
    rlo[threadIdx.x >> 5] = lo;
    rhi[threadIdx.x >> 5] = hi;
    rbad[threadIdx.x >> 5] = nan;
  }
  __syncthreads();
  nan = rbad[0] | rbad[1] | rbad[2] | rbad[3];
  lo = fmin(fmin(rlo[0], rlo[1]), fmin(rlo[2], rlo[3]));
  hi = fmax(fmax(rhi[0], rhi[1]), fmax(rhi[2], rhi[3]));
  const int j = blockIdx.x * 128 + threadIdx.x;
  if (j >= n1) return;
  const double u = x1[j];
  const bool in = u >= lo && u <= hi;
  const int i = in ? locate_sorted(x0, n0, u) : 0;
  const double dx = u - x0[i], w = win ? win[j] : 1.0;
  for (int f = 0; f < nf; ++f) {
    double2 v = make_double2(0, 0);
    if (in) v = spl_eval(y0 + (long long)f * n0, coef + (long long)f * 3 * n0, n0, i, dx);
    if (in && (nan >> 2 * f & 1)) v.x = nan64();
    if (in && (nan >> 2 * f & 2)) v.y = nan64();
    if (win) v = cscale(v, w);
    if (real_part) v.y = 0.0;
    out[(long long)f * n1 + j] = v;
  }
}

// FFTG (usefulsubs.py:2245-2268) of four real fields: F[q] = -(1/N) sum_j f[j] e^{-2 pi i q
// j / N}, one warp per q = 0 .. N / 2 with the wire's table tw[m] = e^{-2 pi i m / N}; F[N - q]
// = conj F[q].
__global__ void __launch_bounds__(64) k_fftg(int n, const double2* tw, const double2* in,
                                             double2* out) {
  pdl_enter();
  const int q = blockIdx.x * 2 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (2 * q > n) return;
  double sr[4] = {0, 0, 0, 0}, si[4] = {0, 0, 0, 0};
  int m = (int)(((long long)q * lane) % n);
  const int step = (int)(((long long)q * 32) % n);
  for (int j = lane; j < n; j += 32) {
    const double2 t = tw[m];
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      const double v = in[(long long)f * n + j].x;
      sr[f] = fma(v, t.x, sr[f]);
      si[f] = fma(v, t.y, si[f]);
    }
    m += step;
    if (m >= n) m -= n;
  }
#pragma unroll
  for (int f = 0; f < 4; ++f)
    for (int o = 16; o > 0; o >>= 1) {
      sr[f] += __shfl_xor_sync(0xffffffffu, sr[f], o);
      si[f] += __shfl_xor_sync(0xffffffffu, si[f], o);
    }
  if (lane < 4) {
    double re = sr[0], im = si[0];
#pragma unroll
    for (int f = 1; f < 4; ++f)
      if (lane == f) {
        re = sr[f];
        im = si[f];
      }
    re = -re / n;
    im = -im / n;
    double2* o = out + (long long)lane * n;
    o[q] = make_double2(re, im);
    if (q > 0 && 2 * q < n) o[n - q] = make_double2(re, -im);
  }
}

// Prop2QW on the context's scratch: the wire-grid part lives in the context's arena;
// the spline coefficients of the caller's grid (12 per point) in a context buffer that
// is allocated on the first call and grown only when a larger grid comes (cudaFree and
// cudaMalloc then wait for the device's pending work); calls of one context are
// ordered on its stream, so they share the scratch.
int launch_prop2qw(SbeCtx* c, int w, const double* RR, int n_rr, const double2* fin,
                   double2* out, cudaStream_t s) {
  const long long need = 12LL * n_rr + spl_bad_elems(n_rr);
  if (need > c->p2q_cap) {
    if (c->p2q_coef && cudaFree(c->p2q_coef) != cudaSuccess)
      return cuda_check(cudaGetLastError(), "prop2qw: release the smaller scratch");
    c->p2q_coef = nullptr;
    c->p2q_cap = 0;
    if (cudaMalloc(&c->p2q_coef, sizeof(double2) * need) != cudaSuccess)
      return fail(SBE_ERR_OOM, "prop2qw scratch");
    c->p2q_cap = need;
  }
  return launch_prop2qw_scratch(c, w, RR, n_rr, fin, out, c->p2q_coef, c->qscr, s);
}

// The same three launches as launch_prop2qw on scratch the caller provides:
// coef holds 12 n_rr + spl_bad_elems(n_rr) and tmp 4 Nr complex values.  Allocates nothing.
int launch_prop2qw_scratch(SbeCtx* c, int w, const double* RR, int n_rr, const double2* fin,
                           double2* out, double2* coef, double2* tmp, cudaStream_t s) {
  const WireDev& W = c->wires[w];
  int* bad = reinterpret_cast<int*>(coef + 12LL * n_rr);
  spline_coefs(n_rr, RR, fin, 4, coef, bad, s);
  launch(k_spline_eval, (W.nr + 127) / 128, 128, 0, s, n_rr, RR, fin, coef, bad, W.nr,
         c->r + W.off_r, 4, c->window + W.off_r, 1, tmp);
  launch(k_fftg, (W.nr / 2 + 2) / 2, 64, 0, s, W.nr, c->twd + W.off_r, tmp, out);
  return cuda_check(cudaGetLastError(), "prop2qw (caller scratch)");
}

// qwoptics.py:760-805 charge renormalisation (Plasmonics).  mode 0: on the wire
// grid (re, rh -> |.| scaled to total); mode 1: on the propagation grid.  One cluster: the
// magnitudes are bound by the FP64 pipe of the blocks' SMs.
__global__ void __cluster_dims__(kCluster, 1, 1) __launch_bounds__(256)
    k_plasmonics(int n, const double* grid, double2* a, double2* b, double* total_io, int mode) {
  pdl_enter();
  const double dx = grid[1] - grid[0];
  const int i0 = blockIdx.x * 256 + threadIdx.x, st = kCluster * 256;
  double A = 0, B = 0;
  for (int j = i0; j < n; j += st) {
    const double x = cabs_d(a[j]), y = cabs_d(b[j]);
    a[j] = make_double2(x, 0);
    b[j] = make_double2(y, 0);
    A += x;
    B += y;
  }
  double total = mode == 0 ? 0.0 : *total_io;
  cluster_sum2(A, B, blockIdx.x * 256 + (threadIdx.x & ~31) < n);
  if (mode == 0) {
    total = (A * dx + B * dx + kQwSmall) / 2.0;
    if (i0 == 0) *total_io = total;
  }
  const double fa = total / (A * dx + kQwSmall), fb = total / (B * dx + kQwSmall);
  for (int j = i0; j < n; j += st) {
    a[j].x *= fa;
    b[j].x *= fb;
  }
}

int launch_qw2prop(SbeCtx* c, int w, const double* RR, int n_rr, const double2* src,
                   double2* out, int plasmonics, cudaStream_t s) {
  // scratch in the context's arena (15 + 5 wire-grid columns and the total)
  const WireDev& W = c->wires[w];
  double2* coef = c->qscr;
  double2* tmp = coef + 15 * (size_t)c->nr_max;
  double* total = reinterpret_cast<double*>(tmp + 5 * (size_t)c->nr_max);
  int* bad = reinterpret_cast<int*>(total + 2);
  cudaMemcpyAsync(tmp, src, sizeof(double2) * 5 * (size_t)W.nr, cudaMemcpyDeviceToDevice, s);
  const double* rw = c->r + W.off_r;
  if (plasmonics)
    launch(k_plasmonics, kCluster, 256, 0, s, W.nr, rw, tmp + 3 * W.nr, tmp + 4 * W.nr, total, 0);
  spline_coefs(W.nr, rw, tmp, 5, coef, bad, s);
  launch(k_spline_eval, (n_rr + 127) / 128, 128, 0, s, W.nr, rw, tmp, coef, bad, n_rr, RR, 5,
         nullptr, 0, out);
  if (plasmonics)
    launch(k_plasmonics, kCluster, 256, 0, s, n_rr, RR, out + 3 * (size_t)n_rr,
           out + 4 * (size_t)n_rr, total, 1);
  return cuda_check(cudaGetLastError(), "qw2prop");
}

}  // namespace sbe

namespace sbe {
void launch_sources_final(SbeCtx* c, const double2* ne, const double2* nh, double2* src,
                          cudaStream_t s) {
  launch(k_src_final, dim3(kCluster, c->nw), 256, 0, s, c->d_wires, -1, c->r, ne, nh, src);
}

void launch_sources_reduce(SbeCtx* c, const double2* ne, const double2* nh, double2* src,
                           cudaStream_t s) {
  launch(k_src_reduce, dim3((c->nr_max + 127) / 128, c->nw), 128, 0, s, c->d_wires, -1, c->expikr,
         c->G, c->tot_kr, c->window, src);
  launch(k_src_final, dim3(kCluster, c->nw), 256, 0, s, c->d_wires, -1, c->r, ne, nh, src);
}
}  // namespace sbe
