"""Measured workloads of the library: what its users run, through the public entry points.

Kinds of case (``case["kind"]``):

* ``solver``: one time step of the drop-in ``SBESolver.QWCalculator`` for every wire, host
  arrays in and out, as the propagation drivers call it (FP64 leapfrog);
* ``functions``: the drop-in pure functions CalcH, dpdt, dCdt, dDdt on device arrays;
* ``rk4``: ``WireContext.rk4_step`` of a batch of wires in a local field (FP64 or mixed);
* ``line``: ``CoupledLine.step``, wires on the 1-D field grid;
* ``grid3``: ``CoupledGrid3.step``, wires along z on the 3-D field grid;
* ``field3``: ``Pstd3D.step``, the 3-D field step alone.

Sizes are those of the benchmark's workloads (``bench.py``), of the tests, and of wires
whose Nk follows from their length as the drop-in solver derives it.  ``exact`` restates
each step in plain torch FP64 (complex128) from the equations.
"""

import math

import numpy as np
import torch

from pulsesuite_gb300 import SBEs, _lib
from pulsesuite_gb300.pstd import CoupledGrid3, CoupledLine, Pstd1D, Pstd3D, SheetSource
from pulsesuite_gb300.wires import WireContext, WireSpec

HBAR = 1.0545718176461565e-34
QE = 1.602176634e-19
EPS0 = 8.8541878188e-12
MU0 = 1.25663706127e-06
ME0 = 9.1093837139e-31
KB = 1.380649e-23
C0 = 299792458.0
EULER = 0.5772156649015329

# GaAs-like wire of the benchmark
MAT = dict(me=0.067 * ME0, mh=0.45 * ME0, gap=1.52 * QE, HO=100e-3 * QE, Delta0=6e-9,
           gam_e=1e12, gam_h=1e12, gam_eh=1e12, epsr=12.9, Oph=36e-3 * QE / HBAR,
           Gph=3e-3 * QE / HBAR)
FLAGS = dict(Optics=True, Excitons=True, EHs=False, Screened=True, Phonon=True, DCTrans=False,
             LF=True, FreePot=False, DiagDph=True, OffDiagDph=True, Recomb=False)
W0 = (MAT["gap"] + 20e-3 * QE) / HBAR          # optical carrier frequency
SWEEP_NK = (64, 96, 128, 192, 256, 384, 512)


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------


def listed():
    return [
        # one wire of 80 nm (Nk = 90) in a propagation run: the smallest call of the drop-in
        dict(name="solver_1x90", kind="solver", nw=1, L=80e-9, nrr=1000, batch=False, temp=77.0),
        # an array of eight 100 nm wires (Nk = 114) stepped in one batch, longer grid
        dict(name="solver_8x114", kind="solver", nw=8, L=100e-9, nrr=4096, batch=True, temp=300.0),
        # the pure functions on arrays a caller holds, at a size that fills no tile
        dict(name="functions_130", kind="functions", nk=130, excitons=True, lf=True),
        # FP64 RK4: the single Nk = 64 wire at 77 K, a medium batch, and large matrices
        dict(name="rk4_fp64_1x64", kind="rk4", nw=1, nk=64, precision="fp64", temp=77.0),
        dict(name="rk4_fp64_8x256", kind="rk4", nw=8, nk=256, precision="fp64", temp=300.0),
        dict(name="rk4_fp64_2x512", kind="rk4", nw=2, nk=512, precision="fp64", temp=300.0),
        # mixed precision: the single wire, where launches count, and a sweep of uneven Nk
        dict(name="rk4_mixed_1x64", kind="rk4", nw=1, nk=64, precision="mixed", temp=77.0),
        dict(name="rk4_mixed_sweep64", kind="rk4", nw=64, nk=0, precision="mixed", temp=300.0),
        # one wire on the 1-D grid, and the benchmark's array of 32 wires
        dict(name="line_mixed_1x256", kind="line", nw=1, nk=256, nx=8192, precision="mixed",
             temp=77.0),
        dict(name="line_mixed_32x512", kind="line", nw=32, nk=512, nx=16384, precision="mixed",
             temp=300.0),
        # wires along z on the 3-D grid (an eighth of the benchmark's wires), and its field step
        dict(name="grid3_mixed_8x1024", kind="grid3", nw=8, nk=1024, nx=256, ny=128, nz=128,
             precision="mixed", temp=77.0),
        dict(name="field3_256x128x128", kind="field3", nx=256, ny=128, nz=128, fp32=True),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(("solver", "functions", "fp64", "fp64", "mixed", "line", "line", "grid3",
                       "field3"))
    temp = float(rng.choice((77.0, 150.0, 300.0)))
    if kind == "solver":
        return dict(kind="solver", nw=rng.randint(1, 8), L=round(_log(rng, 40e-9, 250e-9), 11),
                    nrr=int(_log(rng, 200, 8192)), batch=rng.random() < 0.5, temp=temp)
    if kind == "functions":
        return dict(kind="functions", nk=int(_log(rng, 24, 400)), excitons=rng.random() < 0.8,
                    lf=rng.random() < 0.8)
    if kind == "fp64":
        nk = 2 * int(_log(rng, 16, 257))
        nw = max(1, min(32, int(_log(rng, 1.0, max(1.01, 2.0 * (512.0 / nk) ** 3)))))
        return dict(kind="rk4", nw=nw, nk=nk, precision="fp64", temp=temp)
    if kind == "mixed":
        if rng.random() < 0.3:
            return dict(kind="rk4", nw=rng.randint(8, 64), nk=0, precision="mixed", temp=temp)
        nk = 8 * int(_log(rng, 6, 65))
        return dict(kind="rk4", nw=int(_log(rng, 1, 33)), nk=nk, precision="mixed", temp=temp)
    if kind == "line":
        nx = 2 ** rng.randint(11, 16)
        if rng.random() < 0.25:
            return dict(kind="line", nw=rng.randint(1, 3), nk=2 * int(_log(rng, 16, 129)), nx=nx,
                        precision="fp64", temp=temp)
        return dict(kind="line", nw=int(_log(rng, 1, 17)), nk=8 * int(_log(rng, 6, 65)), nx=nx,
                    precision="mixed", temp=temp)
    dims = [2 ** rng.randint(6, 8), 2 ** rng.randint(5, 7), 2 ** rng.randint(5, 7)]
    if kind == "grid3":
        dims[2] = 2 ** rng.randint(6, 7)
        return dict(kind="grid3", nw=rng.randint(1, 8), nk=8 * int(_log(rng, 8, 97)), nx=dims[0],
                    ny=dims[1], nz=dims[2], precision="mixed", temp=temp)
    return dict(kind="field3", nx=dims[0], ny=dims[1], nz=dims[2], fp32=rng.random() < 0.6)


def wire_length(nk, kmax=3e9):
    """Wire length whose Nk points span |k| <= kmax."""
    return math.pi / (kmax / (nk / 2 - 0.5))


def solver_nk(L):
    """Nk of a wire of length L as the drop-in solver derives it (SBEs.py:4754-4758)."""
    kmax = math.sqrt(1.2 * MAT["gap"] * 2.0 * MAT["me"] / HBAR ** 2)
    return int(math.floor(kmax / (2.0 * math.pi / (2.0 * L))) * 2 + 1) - 1


def case_nks(case):
    """Nk of every wire of an ``rk4``, ``line`` or ``grid3`` case (0: an uneven sweep, its
    wires listed by ascending Nk as the packed layout keeps them)."""
    if case["nk"]:
        return [case["nk"]] * case["nw"]
    g = np.random.default_rng(3)
    p = 1.0 / np.array(SWEEP_NK)
    return sorted(int(v) for v in g.choice(SWEEP_NK, size=case["nw"], p=p / p.sum()))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _cnormal(g, *shape):
    return torch.randn(shape, dtype=torch.complex128, device="cuda", generator=g)


def _state(nk, g):
    """P, C, D of an excited wire: coherences within a Gaussian of the band edge and near
    the diagonal, Hermitian densities over a smooth carrier distribution."""
    k = (torch.arange(nk, dtype=torch.float64, device="cuda") - (nk - 1) / 2.0) / (nk / 2.0)
    env = torch.exp(-(2.5 * k) ** 2)
    near = torch.exp(-((k[:, None] - k[None, :]) * 4.0).abs())
    P = 1e-2 * env[:, None] * env[None, :] * near * _cnormal(g, nk, nk)
    out = [P]
    for n0 in (0.1, 0.08):
        X = 2e-2 * env[:, None] * env[None, :] * near * _cnormal(g, nk, nk)
        X = X + X.conj().T
        X.diagonal().copy_((n0 * env).to(X.dtype) + X.diagonal().real.abs())
        out.append(X)
    return out


def _window_k(nk, L):
    r = np.linspace(-L, L, 2 * nk + 2)
    w = np.exp(-((r / (L / 2.0)) ** 150))
    return r, w


def _wires_inputs(case, seed, coherent=True):
    """Per wire (P, C, D) of the case; coherent=False: P = 0 (the start of a coupled run)."""
    g = _gen(seed)
    out = []
    for nk in case_nks(case):
        P, C, D = _state(nk, g)
        out.append((P if coherent else torch.zeros_like(P), C, D))
    return out


def _local_amplitudes(case, seed):
    r = np.random.default_rng(seed + 1)
    e0 = 10.0 ** r.uniform(6.0, 7.7, case["nw"])
    return e0, 0.1 * e0 * r.uniform(-1.0, 1.0, case["nw"])


def _specs(case):
    return [WireSpec(nk=nk, L=wire_length(nk), temp=case["temp"], wire_index=w + 1,
                     flags=dict(FLAGS), **MAT) for w, nk in enumerate(case_nks(case))]


def _pulse(x, seed, wavelength_k):
    """A travelling pulse on a grid axis: envelope of 1.2 um around a seeded centre."""
    r = np.random.default_rng(seed + 2)
    x0, ph = r.uniform(-0.4e-6, 0.4e-6), r.uniform(0.0, 2.0 * np.pi)
    return np.exp(-((x - x0) / 1.2e-6) ** 2) * np.cos(wavelength_k * x + ph)


def _line_setup(case, seed):
    nx, dx = case["nx"], 10e-9
    x = np.linspace(-(nx - 1) * dx / 2.0, (nx - 1) * dx / 2.0, nx)
    v, eta = C0 / math.sqrt(MAT["epsr"]), math.sqrt(MU0 / (EPS0 * MAT["epsr"]))
    f = 3e7 * _pulse(x, seed, W0 / v)
    E = np.stack([f, 0.3 * f]).astype(complex)
    H = np.stack([f / eta, -0.3 * f / eta]).astype(complex)
    return dict(dx=dx, dt=0.05e-15, n_abc=min(128, nx // 16), abc=0.05, E=E, H=H,
                Ex=np.zeros(nx, complex), src=nx // 4, E0=5e7, tau=50e-15, t0=-20e-15,
                wx=(np.arange(case["nw"]) - (case["nw"] - 1) / 2.0) * 100e-9)


def _grid3_setup(case, seed):
    n, d = (case["nx"], case["ny"], case["nz"]), 20e-9
    ax = [np.linspace(-(m - 1) * d / 2.0, (m - 1) * d / 2.0, m) for m in n]
    v, eta = C0 / math.sqrt(MAT["epsr"]), math.sqrt(MU0 / (EPS0 * MAT["epsr"]))
    beam = np.exp(-(ax[1][:, None] ** 2 + ax[2][None, :] ** 2) / 1e-6 ** 2)
    f = torch.as_tensor(2e7 * _pulse(ax[0], seed, W0 / v)).cuda()[:, None, None] * \
        torch.as_tensor(beam).cuda()[None]
    E = torch.zeros((3,) + n, dtype=torch.complex128, device="cuda")
    H = torch.zeros_like(E)
    E[1], H[2] = f, f / eta
    r = np.random.default_rng(4)
    xy = [(float(r.uniform(-0.3, 0.3) * n[0] * d), float(r.uniform(-0.3, 0.3) * n[1] * d))
          for _ in range(case.get("nw", 0))]
    return dict(n=n, d=d, dt=0.02e-15, n_abc=tuple(max(2, m // 16) for m in n), abc=0.05, E=E,
                H=H, xy=xy, src=n[0] // 8, E0=2e7, tau=80e-15, t0=-20e-15, waist=1e-6, gate=5e-9)


def _solver_setup(case, seed):
    r = np.random.default_rng(seed)
    nk, nw, nrr = solver_nk(case["L"]), case["nw"], case["nrr"]
    half = 2.5 * case["L"]
    rr = np.linspace(-half, half, nrr)
    g = _gen(seed)
    st = [[m.cpu().numpy() for m in _state(nk, g)] for _ in range(nw)]
    fields = []
    for _ in range(nw):
        env = np.exp(-(rr / half) ** 2)
        a = 2e7 * r.uniform(0.5, 1.0, 3)
        ph = r.uniform(0, 2 * np.pi, 3)
        fields.append([(a[c] * env * np.cos(2e6 * rr + ph[c])).astype(complex) for c in range(3)]
                      + [np.zeros(nrr, complex)])
    return nk, rr, st, fields


def _function_inputs(case, seed):
    nk = case["nk"]
    g = _gen(seed)
    P, C, D = _state(nk, g)
    k = (torch.arange(nk, dtype=torch.float64, device="cuda") - (nk - 1) / 2.0) * (6e9 / nk)
    Ee, Eh = HBAR ** 2 * k ** 2 / (2 * MAT["me"]), HBAR ** 2 * k ** 2 / (2 * MAT["mh"])
    dist = torch.arange(nk, dtype=torch.float64, device="cuda")
    v = 5e-22 * torch.log(1.0 + 20.0 / (dist + 0.5))
    VC = torch.zeros((nk, nk, 3), dtype=torch.float64, device="cuda")
    VC[:, 0, :] = v[:, None] * torch.tensor([1.0, 1.1, 0.9], dtype=torch.float64, device="cuda")
    Meh = 3e-21 * torch.exp(-((k[:, None] - k[None, :]) / 4e8) ** 2) * (1.0 + 0.1 * _cnormal(g, nk, nk))
    gam = 1e12 * (1.0 + torch.rand(2, nk, dtype=torch.float64, device="cuda", generator=g))
    OffP = 1e-24 * _cnormal(g, nk, nk)
    return P, C, D, Ee, Eh, VC, Meh, gam[0].contiguous(), gam[1].contiguous(), OffP


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------


def _prec(case):
    return _lib.PREC_MIXED if case["precision"] == "mixed" else _lib.PREC_FP64


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=dict(case))
    if kind == "solver":
        nk, rr, st, fields = _solver_setup(case, seed)
        params = dict(MAT, L=case["L"], Edc=0.0, jmax=1000, ntmax=100000)
        sv = SBEs.SBESolver(None, rr, 0.0, 2e7, 8e-7, case["nw"], True, params=params,
                            flags=dict(FLAGS), temp=case["temp"], batch=case["batch"])
        sv.write_info = False      # the per-step text diagnostics grow a file on disk
        for i, names in enumerate((("YY2", "YY3"), ("CC2", "CC3"), ("DD2", "DD3"))):
            lev = np.stack([w[i] for w in st], axis=2)
            for n in names:
                setattr(sv, n, lev)
        s.update(solver=sv, rr=rr, fields=fields,
                 outs=[[np.zeros(len(rr), complex) for _ in range(4)] for _ in range(case["nw"])])
    elif kind == "functions":
        (s["P"], s["C"], s["D"], s["Ee"], s["Eh"], s["VC"], s["Meh"], s["ge"], s["gh"],
         s["OffP"]) = _function_inputs(case, seed)
        s["H"] = [torch.empty_like(s["P"]) for _ in range(3)]
        s["Z"] = torch.zeros_like(s["P"])
    elif kind == "field3":
        q = _grid3_setup(case, seed)
        s["grid"] = Pstd3D(q["n"], (q["d"],) * 3, MAT["epsr"], n_abc=q["n_abc"],
                           abc_strength=q["abc"], fp32_work=case["fp32"])
        g = _gen(seed)
        s.update(E=q["E"], H=q["H"], dt=q["dt"])
        s["E"][0] += 1e5 * _cnormal(g, *q["n"])
        s["J"] = 1e9 * _cnormal(g, 3, *q["n"])
    else:
        ctx = WireContext(_specs(case))
        mats = _wires_inputs(case, seed, coherent=(kind == "rk4"))
        s["ctx"] = ctx
        s["P"], s["C"], s["D"] = (ctx.pack([m[i] for m in mats]) for i in range(3))
        if kind == "rk4":
            e0, de = _local_amplitudes(case, seed)
            s["Ek"], s["dEk"] = ctx.local_field(e0, de)
            s["src"] = ctx.zeros_r(5)
        elif kind == "line":
            q = _line_setup(case, seed)
            s["grid"] = Pstd1D(case["nx"], q["dx"], MAT["epsr"], n_abc=q["n_abc"],
                               abc_strength=q["abc"])
            s["line"] = CoupledLine(ctx, s["grid"], q["wx"],
                                    source=SheetSource(q["src"], q["E0"], q["tau"], W0, 0.0),
                                    t0=q["t0"])
            s.update(dt=q["dt"], E=torch.as_tensor(q["E"]).cuda(), H=torch.as_tensor(q["H"]).cuda(),
                     Ex=torch.as_tensor(q["Ex"]).cuda())
        else:
            q = _grid3_setup(case, seed)
            s["grid"] = Pstd3D(q["n"], (q["d"],) * 3, MAT["epsr"], n_abc=q["n_abc"],
                               abc_strength=q["abc"], fp32_work=True)
            s["line"] = CoupledGrid3(ctx, s["grid"], q["xy"],
                                     source=SheetSource(q["src"], q["E0"], q["tau"], W0, 0.0),
                                     pol=1, waist=q["waist"], gate=q["gate"], t0=q["t0"])
            s.update(dt=q["dt"], E=q["E"], H=q["H"])
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "solver":
        for w in range(1, case["nw"] + 1):
            f, o = s["fields"][w - 1], s["outs"][w - 1]
            s["solver"].QWCalculator(f[0], f[1], f[2], f[3], s["rr"], None, 0.05e-15, w, o[0], o[1],
                                     o[2], o[3], [False], [False])
        return s["outs"]
    if kind == "functions":
        H = s["H"]
        SBEs.calc_h(s["Meh"], s["Z"], s["Z"], s["C"], s["D"], s["P"], s["VC"], *H, s["Ee"], s["Eh"],
                    MAT["gap"], case["excitons"], case["lf"], False)
        dP = SBEs.dpdt(s["C"], s["D"], s["P"], *H, s["ge"], s["gh"], s["OffP"])
        dC = SBEs.dCdt(s["C"], s["D"], s["P"], *H, s["ge"], s["gh"], s["OffP"])
        dD = SBEs.dDdt(s["C"], s["D"], s["P"], *H, s["ge"], s["gh"], s["OffP"])
        return dict(H=H, dP=dP, dC=dC, dD=dD)
    if kind == "rk4":
        s["ctx"].rk4_step(s["P"], s["C"], s["D"], s["Ek"], s["dEk"], 0.1e-15, s["src"], _prec(case))
        return dict(P=s["P"], C=s["C"], D=s["D"], src=s["src"])
    if kind == "line":
        s["line"].step(s["P"], s["C"], s["D"], s["E"], s["H"], s["Ex"], s["dt"], _prec(case))
        # the view is the line's own memory: a caller that keeps the sources copies them
        return dict(P=s["P"], C=s["C"], D=s["D"], E=s["E"], H=s["H"], Ex=s["Ex"],
                    src=s["line"].view("src").clone())
    if kind == "grid3":
        s["line"].step(s["P"], s["C"], s["D"], s["E"], s["H"], s["dt"], _prec(case))
        return dict(P=s["P"], C=s["C"], D=s["D"], E=s["E"], H=s["H"],
                    src=s["line"].view("src").clone())
    s["grid"].step(s["E"], s["H"], s["J"], s["dt"])
    return dict(E=s["E"], H=s["H"])


def _rhs_work(nk):
    """Flops of one RHS evaluation: 12 complex products, three exchange sums over the band."""
    return 96.0 * nk ** 3 + 8.0 * nk ** 3


def _dephasing_work(nk):
    """The Lorentzian sums of both species, q and -q, a-a and a-b: about Nk^3 / 3 (q, k, p)
    triples each, a Lorentzian and two sums per triple."""
    return 4.0 * (nk ** 3 / 3.0) * 10.0


def work(case):
    kind = case["kind"]
    if kind == "solver":
        nk = solver_nk(case["L"])
        nr = 2 * nk + 2
        per = _rhs_work(nk) + _dephasing_work(nk) + 24.0 * nk * nk * nr
        return dict(bytes=case["nw"] * (15 * 16.0 * nk * nk + 8 * 16.0 * case["nrr"]),
                    flops=case["nw"] * per)
    if kind == "functions":
        return dict(bytes=14 * 16.0 * case["nk"] ** 2 + 24.0 * case["nk"] ** 2,
                    flops=_rhs_work(case["nk"]))
    if kind == "field3":
        n = case["nx"] * case["ny"] * case["nz"]
        return dict(bytes=240.0 * n, flops=12 * 2 * 5.0 * n * math.log2(n))
    b = f = 0.0
    for nk in case_nks(case):
        b += 6 * 16.0 * nk * nk + 11 * 16.0 * (2 * nk + 2)
        f += 4 * _rhs_work(nk) + _dephasing_work(nk) + 24.0 * nk * nk * (2 * nk + 2)
    if kind == "line":
        b += 10 * 16.0 * case["nx"]
        f += 8 * 5.0 * case["nx"] * math.log2(case["nx"])
    elif kind == "grid3":
        n = case["nx"] * case["ny"] * case["nz"]
        b += 192.0 * n
        f += 12 * 2 * 5.0 * n * math.log2(n)
    return dict(bytes=b, flops=f)


# ---------------------------------------------------------------------------
# the same steps in plain torch FP64
# ---------------------------------------------------------------------------


def _dev(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda", dtype=dtype)


def _k0_truncated(x):
    """The K0 of the V(q) tables (coulomb.py:39-66)."""
    ser = (x >= 1e-10) & (x < 2.0)
    xs = torch.where(ser, x, torch.ones_like(x))
    res = -torch.log(0.5 * xs) - EULER
    term, live = torch.ones_like(xs), torch.ones_like(xs, dtype=torch.bool)
    for k in range(1, 20):
        term = torch.where(live, term * 0.25 * xs * xs / (k * k), term)
        res = torch.where(live, res + term * (1.0 / k - EULER), res)
        live = live & (term.abs() >= 1e-15)
    asy = torch.sqrt(math.pi / (2.0 * x.clamp_min(1e-10))) * torch.exp(-x)
    out = torch.where(ser, res, torch.where(x <= 100.0, asy, torch.zeros_like(x)))
    return torch.where(x < 1e-10, torch.full_like(x, 23.0), out)


def _dfact(n):
    return 1.0 if n <= 1 else n * _dfact(n - 2)


def _k0(x):
    """The K0 of the Chi1D tables (usefulsubs.py:1649-1800)."""
    if x > 100.0:
        return 0.0
    if x <= 9.0:
        cs, ct, w0, cr, cw = 0.0, -math.log(0.5 * x) - EULER, 0.0, 1.0, 0.0
        for k in range(1, 51):
            w0 += 1.0 / k
            cr = 0.25 * cr * (1.0 / (k * k)) * (x * x)
            cs += cr * (w0 + ct)
            if abs((cs - cw) / cs) < 1e-15:
                break
            cw = cs
        return ct + cs
    s = 1.0 + sum(_dfact(2 * k - 1) ** 3 / (_dfact(2 * k) * 4.0 ** k) * x ** (-2 * k)
                  for k in range(1, 11))
    if x <= 18.0:
        i0, cr = 1.0, 1.0
        for k in range(1, 51):
            cr = 0.25 * cr * (x * x) / (k * k)
            i0 += cr
            if abs(cr / i0) < 1e-15:
                break
    else:
        n = 12 if x < 35.0 else (9 if x < 50.0 else 7)
        i0 = math.exp(x) / math.sqrt(2.0 * math.pi * x) * (1.0 + sum(
            _dfact(2 * k - 1) ** 2 / (math.factorial(k) * 8.0 ** k) * x ** -k
            for k in range(1, n + 1)))
    return 0.5 / x * s / i0


class _Tables:
    """Grid, Coulomb, phonon and dephasing tables of a wire (Nk, L, temperature)."""

    def __init__(self, nk, L, temp):
        self.nk, self.L, self.nr = nk, L, 2 * nk + 2
        m, dk = MAT, math.pi / L
        self.kr = kr = dk * (np.arange(nk) - (nk - 1) // 2 - 0.5)
        self.dk = dk
        self.r, win = _window_k(nk, L)
        self.win = _dev(win)
        self.Ee, self.Eh = (_dev(HBAR ** 2 * kr ** 2 / (2 * m[x])) for x in ("me", "mh"))
        ae, ah = math.sqrt(m["me"] * m["HO"]) / HBAR, math.sqrt(m["mh"] * m["HO"]) / HBAR
        self.dcv = math.sqrt((QE * HBAR) ** 2 / (6.0 * ME0 * m["gap"]) * (ME0 / m["me"] - 1.0))
        self.ehint = math.sqrt(2.0 * ae * ah / (ae * ae + ah * ah))
        self.area = math.sqrt(2.0 * math.pi) / math.sqrt(ae * ae + ah * ah) * m["Delta0"]
        n1, n2 = self.nr // 4, 3 * self.nr // 4
        y = _dev(self.r[n1:n2 + 1])
        ny = len(y)
        off = (torch.arange(ny, device="cuda")[:, None] - torch.arange(ny, device="cuda")).reshape(-1)
        dist = torch.sqrt((y - y[0]) ** 2 + m["Delta0"] ** 2)
        q = _dev(np.arange(nk) * dk)
        pref = QE ** 2 / (2 * math.pi * EPS0 * m["epsr"] * L)
        self.v0 = []
        for a1, a2 in ((ae, ah), (ae, ae), (ah, ah)):          # eh, ee, hh
            pair = torch.exp(-(a1 * y[:, None]) ** 2 - (a2 * y[None, :]) ** 2).reshape(-1)
            cor = torch.zeros(ny, dtype=torch.float64, device="cuda").index_add_(0, off.abs(), pair)
            kd = _k0_truncated(torch.clamp_min(q, (a1 + a2) / 4.0)[:, None] * dist[None, :])
            mult = a1 * a2 / math.pi * (self.r[1] - self.r[0]) ** 2
            self.v0.append(pref * mult * (kd @ cor))
        dif = np.abs(kr - kr[0])
        sc = QE ** 2 / (2 * math.pi * EPS0 * m["epsr"] * HBAR ** 2)
        self.q, self.chi = [], []
        for mass, a in ((m["me"], ae), (m["mh"], ah)):
            qa = np.maximum(dif, a / 2.0)
            R = math.sqrt((2.0 / a) ** 2 + m["Delta0"] ** 2)
            self.q.append(_dev(qa))
            self.chi.append(_dev([mass * _k0(v * R) / v * sc for v in qa]))
        self.nmax = min(ae, ah) / 2.0 / math.pi * 0.99
        n0 = 1.0 / (math.exp(HBAR * m["Oph"] / KB / temp) - 1.0)
        hO, hG = HBAR * m["Oph"], HBAR * m["Gph"]
        self.ph = []
        for e in (self.Ee, self.Eh):
            d = e[:, None] - e[None, :]
            t = n0 / ((d - hO) ** 2 + hG ** 2) + (n0 + 1.0) / ((d + hO) ** 2 + hG ** 2)
            t = t * 2.0 * m["Gph"]
            t.diagonal().zero_()
            self.ph.append(t)
        self.vscale = hO * m["epsr"] * (1.0 / 8.2 - 1.0 / 10.0)
        k, i = _dev(kr), torch.arange(nk, device="cuda")
        kmax, kmin = kr[-1] + (kr[1] - kr[0]), kr[0] - (kr[1] - kr[0])

        def idx(v):
            return torch.round(v.clamp(kmin, kmax) / (kr[1] - kr[0])).long() + (nk - 1) // 2
        K, Q = k[:, None], k[None, :]
        self.kpq, self.kmq = idx(K + Q), idx(K - Q)
        me, mh = m["me"], m["mh"]
        kp, kn = ((me + mh) * Q - 2 * mh * K) / 2.0 / me, ((me + mh) * Q - 2 * me * K) / 2.0 / mh
        self.part = ((idx(kp), idx(kp - Q)), (idx(kn), idx(kn - Q)))
        self.x = [ma / HBAR ** 2 * k.abs() / (k.abs() + (kr[1] - kr[0]) * 1e-5) ** 2 / (kr[1] - kr[0])
                  for ma in (me, mh)]
        self.iq = torch.round((k / (kr[1] - kr[0])).abs()).long()
        self.dif = (i[:, None] - i[None, :])
        self.E = torch.exp(1j * (k[:, None] * _dev(self.r)[None, :]))
        # shear: column d + Nk - 1 holds the diagonal (j, j + d)
        jj = i[:, None] + torch.arange(-(nk - 1), nk, device="cuda")[None, :]
        self.sh_ok, self.sh_j = (jj >= 0) & (jj < nk), jj.clamp(0, nk - 1)

    def screen(self, ne, nh):
        n = min(float((ne.real + nh.real).sum()) / 2.0 / self.L, self.nmax)
        e = 1.0
        for q, c in zip(self.q, self.chi):
            e = e - c * 2 * torch.log(((q - math.pi * n) / (q + n)).abs())
        return e, [v / e for v in self.v0]

    def gammas(self, ne, nh, v):
        def pick(a, i):
            ok = (i >= 0) & (i < self.nk)
            return a[i.clamp(0, self.nk - 1)], ok
        out = []
        for s, (a, b) in enumerate(((ne.real, nh.real), (nh.real, ne.real))):
            vaa2, veh2 = v[1 + s][self.iq] ** 2, v[0][self.iq] ** 2
            n, ok = pick(a, self.kpq)
            t = torch.where(ok, vaa2 * n * (1 - n) * self.x[s].abs(), 0.0 * n)
            (n2, o2), (n1, o1), (n3, o3) = (pick(b, self.part[s][0]), pick(b, self.part[s][1]),
                                            pick(a, self.kmq))
            u = veh2 * (n1 * (1 - n2) * n3 + (1 - n1) * n2 * (1 - n3)) * self.x[1 - s].abs()
            out.append(math.pi / HBAR * (t + torch.where(o1 & o2 & o3, u, 0.0 * u)).sum(1))
        return out

    def exchange(self, v, X):
        """sum_q v(|q|) X[k1 + q][k2 + q], q != 0."""
        t = v[self.dif.abs()].clone()
        t.diagonal().zero_()
        j = torch.arange(self.nk, device="cuda")
        S = torch.where(self.sh_ok, X[j[:, None], self.sh_j], torch.zeros((), dtype=X.dtype, device="cuda"))
        R = t.to(X.dtype) @ S
        return R[j[:, None], self.nk - 1 - self.dif]

    def traces(self, X):
        """tr_d = sum_k X[k][k + d] at index d + Nk - 1."""
        j = torch.arange(self.nk, device="cuda")
        return torch.where(self.sh_ok, X[j[:, None], self.sh_j],
                           torch.zeros((), dtype=X.dtype, device="cuda")).sum(0)


def _dephasing(nk, L, occ, v):
    """De, Dh contraction matrices (B, A) of wires that share Nk: occ, v per wire."""
    t = _Tables.cache[nk, L]
    g = (MAT["gam_eh"], MAT["gam_e"], MAT["gam_h"])
    out = [[], []]
    nw = len(occ)
    for s in range(2):
        na = torch.stack([o[s].abs() for o in occ], 1)
        nb = torch.stack([o[1 - s].abs() for o in occ], 1)
        vaa = torch.stack([x[1 + s] for x in v], 1) ** 2
        vab = torch.stack([x[0] for x in v], 1) ** 2
        Ea, Eb = (t.Ee, t.Eh) if s == 0 else (t.Eh, t.Ee)
        ba, bb = HBAR * g[s], HBAR * g[2]
        M = torch.zeros((nw, nk, nk), dtype=torch.float64, device="cuda")
        for q in range(-(nk - 1), nk):
            if q == 0:
                continue
            k = slice(max(0, -q), nk - max(0, q))
            kq = slice(max(0, q), nk + min(0, q))
            tot = 0.0
            lo, hi = max(q + 1, 0), min(q + nk, nk)
            for E2, n2, pa, pb, b, vv in (
                    (Ea, na, slice(lo - q, hi - q), slice(lo, hi), ba, vaa),
                    (Eb, nb, slice(max(0, -q) + q, nk - max(0, q) + q), slice(max(0, -q), nk - max(0, q)),
                     bb, vab)):
                if pb.stop <= pb.start:
                    continue
                u = (Ea[kq] - Ea[k])[:, None] + (E2[pa] - E2[pb])[None, :]
                lr = (b / math.pi) / (u * u + b * b)
                w1, w2 = n2[pa] * (1 - n2[pb]), (1 - n2[pa]) * n2[pb]
                tot = tot + vv[abs(q)] * ((lr @ w1) * (1 - na[k]) + (lr @ w2) * na[k])
            if torch.is_tensor(tot):
                M.diagonal(q, 1, 2).copy_((tot * math.pi / HBAR).T)
        out[s] = M
    return out            # [from De, from Dh], [wire][row][j]


_Tables.cache = {}


def _tables(nk, L, temp):
    if (nk, L) not in _Tables.cache or _Tables.cache[nk, L].temp != temp:
        while len(_Tables.cache) > 12:
            _Tables.cache.pop(next(iter(_Tables.cache)))
        _Tables.cache[nk, L] = _Tables(nk, L, temp)
        _Tables.cache[nk, L].temp = temp
    return _Tables.cache[nk, L]


def _yw(w):
    return 1.0 if ((w - 1) // 2) % 2 == 0 else -1.0


def _dipole(t, Ek, w):
    q = t.dif % t.nr
    sg = 1.0 - 2.0 * (torch.arange(t.nk, device="cuda") % 2).double()
    return -t.ehint * t.dcv * (sg[None, :] * Ek[0][q] + _yw(w) * Ek[1][q]
                               - (1.0 if w % 2 == 0 else -1.0) * Ek[2][q])


def _hamiltonian(t, Meh, P, C, D, v, Ee, Eh, excitons=True, lf=True):
    dg = torch.diag_embed
    Heh, Hee, Hhh = Meh.clone(), dg(Ee + MAT["gap"]).to(P.dtype), dg(Eh).to(P.dtype)
    if not excitons:
        return Heh, Hee, Hhh
    Heh = Heh + t.exchange(v[0], P.T)
    if lf:
        Hee = Hee - t.exchange(v[1], C.T)
        Hhh = Hhh - t.exchange(v[2], D.T)
        tc, td = t.traces(C), t.traces(D)
        d, n, o = t.dif, t.nk - 1, (t.dif != 0)
        Hee = Hee + o * (v[1][d.abs()] * tc[d + n] - v[0][d.abs()] * td[n - d])
        Hhh = Hhh + o * (v[2][d.abs()] * td[d + n] - v[0][d.abs()] * tc[n - d])
    else:
        m = t.dif.abs()
        off = (t.dif != 0).double()
        Hee = Hee - dg((v[1][m] * off).to(P.dtype) @ C.diagonal())
        Hhh = Hhh - dg((v[2][m] * off).to(P.dtype) @ D.diagonal())
    return Heh, Hee, Hhh


def _rhs(P, C, D, Heh, Hee, Hhh, ge, gh, offp):
    ih = 1j * HBAR
    dP = (Hhh @ P + P @ Hee.T - Heh.T @ C - (Heh @ D).T + Heh.T
          - ih * (ge[None, :] + gh[:, None]) * P + offp) / ih
    dC = (C @ Hee.T - Hee.T @ C + P.conj().T @ Heh.T - Heh.conj() @ P) / ih
    dD = (D @ Hhh.T - Hhh.T @ D + P.conj() @ Heh - Heh.conj().T @ P.T) / ih
    return dP, dC, dD


def _frozen(ts, Cs, Ds):
    """Occupation-dependent coefficients of every wire (evaluated once per step)."""
    occ = [(C.diagonal().clone(), D.diagonal().clone()) for C, D in zip(Cs, Ds)]
    scr = [t.screen(*o) for t, o in zip(ts, occ)]
    co = [dict(eps=e, v=v, gam=t.gammas(*o, v)) for t, o, (e, v) in zip(ts, occ, scr)]
    for nk in sorted({t.nk for t in ts}):
        ws = [i for i, t in enumerate(ts) if t.nk == nk]
        B, A = _dephasing(nk, ts[ws[0]].L, [occ[i] for i in ws], [co[i]["v"] for i in ws])
        for n, i in enumerate(ws):
            co[i].update(A=A[n].to(torch.complex128), B=B[n].to(torch.complex128))
    return co


def _relax(t, c, C, D, dt):
    out = []
    for s, X in enumerate((C, D)):
        n = X.diagonal().clone()
        d = t.dif if s == 0 else -t.dif                   # nonzero for k >= i (e), i >= k (h)
        vep = torch.where(d >= 0, c["v"][1 + s][d.abs()] / c["eps"][d.abs()] * t.vscale, 0.0 * d)
        win = (vep * t.ph[s]) @ n.real
        wout = (vep * t.ph[s].T) @ (1.0 - n.real)
        W = win + wout
        out.append(torch.exp(-W * dt) * ((-1 + torch.exp(W * dt) + n) * win + n * wout) / (W + 1e-200))
    ne, nh = out[0].abs(), out[1].abs()
    tot = (ne.sum() + nh.sum()) / 2.0
    ne, nh = ne * tot / (ne.sum() + 1e-200), nh * tot / (nh.sum() + 1e-200)
    C.diagonal().copy_(ne.to(C.dtype))
    D.diagonal().copy_(nh.to(D.dtype))
    return ne, nh


def _sources(t, P, C, D, ne, nh, w):
    """Real-space Px, Py, Pz, re, rh (5, Nr)."""
    E, Ec = t.E, t.E.conj()
    G = (Ec * (P @ E)).real
    sg = 1.0 - 2.0 * (torch.arange(t.nk, device="cuda") % 2).double()
    f = 2 * t.ehint / t.area / t.L * t.dcv * t.win
    sx, sy = (sg[:, None] * G).sum(0) * f, G.sum(0) * f
    out = [sx, sy * _yw(w), -sy * (1.0 if w % 2 == 0 else -1.0)]
    dr = t.r[1] - t.r[0]
    for X, n in ((C, ne), (D.conj(), nh)):
        x = (Ec * (X @ E)).sum(0) * t.win / (2.0 * t.L)
        x = x - (x[:10].sum() + x[-10:].sum()).real / 20.0
        x = x * ((n.sum() + 1e-50) / (x.abs().sum() * dr + 1e-100))
        out.append(2.0 * QE * x / t.area * t.ehint)
    return torch.stack([o.to(torch.complex128) for o in out])


def _rk4(ts, mats, Ek, dEk, dt):
    """One RK4 step of every wire: (P, C, D, sources) per wire."""
    co = _frozen(ts, [m[1] for m in mats], [m[2] for m in mats])
    out = []
    for w, (t, c, X) in enumerate(zip(ts, co, mats)):
        def f(S, frac):
            H = _hamiltonian(t, _dipole(t, Ek[w] + frac * dEk[w], w + 1), *S, c["v"], t.Ee, t.Eh)
            return _rhs(*S, *H, *c["gam"], 1j * HBAR * (c["A"] @ S[0] + S[0] @ c["B"].T))
        k1 = f(X, 0.0)
        k2 = f([x + 0.5 * dt * k for x, k in zip(X, k1)], 0.5)
        k3 = f([x + 0.5 * dt * k for x, k in zip(X, k2)], 0.5)
        k4 = f([x + dt * k for x, k in zip(X, k3)], 1.0)
        P, C, D = (x + dt / 6.0 * (a + 2.0 * b + 2.0 * d + e)
                   for x, a, b, d, e in zip(X, k1, k2, k3, k4))
        ne, nh = _relax(t, c, C, D, dt)
        out.append((P, C, D, _sources(t, P, C, D, ne, nh, w + 1)))
    return out


def _fftg(f):
    return -torch.fft.fft(f) / f.shape[-1]


def _spline(x, y):
    """Forsythe-Malcolm-Moler cubic spline (spliner.py:1329-1394) of the rows of y."""
    y = np.asarray(y)
    n, h = len(x), np.diff(x)
    dy = np.diff(y, axis=1) / h
    c = np.zeros(y.shape, complex)
    c[:, 1:-1] = dy[:, 1:] - dy[:, :-1]
    b = np.empty(n)
    b[0], b[-1], b[1:-1] = -h[0], -h[-1], 2.0 * (h[:-1] + h[1:])
    c[:, 0] = (c[:, 2] / (x[3] - x[1]) - c[:, 1] / (x[2] - x[0])) * h[0] ** 2 / (x[3] - x[0])
    c[:, -1] = -(c[:, -2] / (x[-1] - x[-3]) - c[:, -3] / (x[-2] - x[-4])) * h[-1] ** 2 / (x[-1] - x[-4])
    c = np.ascontiguousarray(c.T)
    for i in range(1, n):
        f = h[i - 1] / b[i - 1]
        b[i] -= f * h[i - 1]
        c[i] -= f * c[i - 1]
    c[-1] /= b[-1]
    for i in range(n - 2, -1, -1):
        c[i] = (c[i] - h[i] * c[i + 1]) / b[i]
    c = c.T
    B = np.concatenate([dy - h * (c[:, 1:] + 2.0 * c[:, :-1]),
                        (dy[:, -1] + h[-1] * (c[:, -2] + 2.0 * c[:, -1]))[:, None]], axis=1)
    d = np.diff(c, axis=1) / h
    return B, 3.0 * c, np.concatenate([d, d[:, -1:]], axis=1)


def _resample(x, y, u, coef=None):
    b, c, d = coef if coef is not None else _spline(x, y)
    j = np.clip(np.searchsorted(x, u, side="right") - 1, 0, len(x) - 1)
    s = u - x[j]
    v = y[:, j] + s * (b[:, j] + s * (c[:, j] + s * d[:, j]))
    return np.where((u >= x[0]) & (u <= x[-1]), v, 0.0)


def _to_wire(t, vals):
    """Windowed real fields on the wire grid to wire k space."""
    v = torch.as_tensor(vals, device="cuda") * t.win
    return _fftg(v.real.to(torch.complex128))


def _exact_solver(case, seed):
    nk, rr, st, fields = _solver_setup(case, seed)
    t = _tables(nk, case["L"], case["temp"])
    dt = 0.05e-15
    mats = [[_dev(m, torch.complex128) for m in w] for w in st]
    co = _frozen([t] * case["nw"], [m[1] for m in mats], [m[2] for m in mats])
    outs = []
    for w, (c, X, f) in enumerate(zip(co, mats, fields)):
        Ek = _to_wire(t, _resample(rr, np.stack(f), t.r))
        H = _hamiltonian(t, _dipole(t, Ek, w + 1), *X, c["v"], t.Ee, t.Eh)
        k = _rhs(*X, *H, *c["gam"], 1j * HBAR * (c["A"] @ X[0] + X[0] @ c["B"].T))
        P, C, D = (x + 2.0 * dt * d for x, d in zip(X, k))
        ne, nh = _relax(t, c, C, D, dt)
        s = _sources(t, P, C, D, ne, nh, w + 1).cpu().numpy()
        dr, dR = t.r[1] - t.r[0], rr[1] - rr[0]
        s[3:] = np.abs(s[3:])
        tot = (s[3].sum() * dr + s[4].sum() * dr + 1e-100) / 2.0
        s[3:] *= (tot / (s[3:].sum(1) * dr + 1e-100))[:, None]
        g = _resample(t.r, s, rr)
        g[3:] = np.abs(g[3:])
        g[3:] *= (tot / (g[3:].sum(1) * dR + 1e-100))[:, None]
        outs.append([g[0], g[1], g[2], g[4] - g[3]])
    return outs


def _exact_functions(case, seed):
    P, C, D, Ee, Eh, VC, Meh, ge, gh, OffP = _function_inputs(case, seed)
    nk = case["nk"]
    t = object.__new__(_Tables)
    i = torch.arange(nk, device="cuda")
    t.nk, t.dif = nk, i[:, None] - i[None, :]
    jj = i[:, None] + torch.arange(-(nk - 1), nk, device="cuda")[None, :]
    t.sh_ok, t.sh_j = (jj >= 0) & (jj < nk), jj.clamp(0, nk - 1)
    H = _hamiltonian(t, Meh, P, C, D, [VC[:, 0, n] for n in range(3)], Ee, Eh, case["excitons"],
                     case["lf"])
    dP, dC, dD = _rhs(P, C, D, *H, ge, gh, OffP)
    return dict(H=list(H), dP=dP, dC=dC, dD=dD)


def _packed(parts):
    """Per-wire blocks as the packed layout holds them."""
    return torch.cat([p.reshape(-1) for p in parts])


def _case_tables(case):
    return [_tables(nk, wire_length(nk), case["temp"]) for nk in case_nks(case)]


def _exact_rk4(case, seed):
    ts, mats = _case_tables(case), _wires_inputs(case, seed)
    e0, de = _local_amplitudes(case, seed)
    Ek, dEk = [], []
    for t, a, b in zip(ts, e0, de):
        wk = _fftg(t.win.to(torch.complex128))
        Ek.append(torch.stack([0 * wk, a * wk, 0 * wk]))
        dEk.append(torch.stack([0 * wk, b * wk, 0 * wk]))
    o = _rk4(ts, mats, Ek, dEk, 0.1e-15)
    return dict(P=_packed([x[0] for x in o]), C=_packed([x[1] for x in o]),
                D=_packed([x[2] for x in o]), src=_packed([x[3] for x in o]))


def _fft_q(n, d):
    i = np.arange(n)
    return np.where(i <= n // 2, i, i - n) * (2.0 * np.pi / (n * d))


def _mask(n, na, strength):
    j = np.arange(n)
    s = np.maximum(0, na - np.minimum(j, n - 1 - j)) / max(na, 1)
    return np.exp(-strength * s * s)


def _sheet(q, dx, dt):
    eta = math.sqrt(MU0 / (EPS0 * MAT["epsr"]))
    th = q["t0"] + 0.5 * dt
    return -2.0 * q["E0"] / (eta * dx) * math.exp(-(th / q["tau"]) ** 2) * math.cos(W0 * th)


def _exact_line(case, seed):
    q = _line_setup(case, seed)
    ts, mats = _case_tables(case), _wires_inputs(case, seed, coherent=False)
    nx, dx, dt = case["nx"], q["dx"], q["dt"]
    x = np.linspace(-(nx - 1) * dx / 2.0, (nx - 1) * dx / 2.0, nx)
    qx = _dev(_fft_q(nx, dx))
    mask = _dev(_mask(nx, q["n_abc"], q["abc"]))
    y = np.stack([q["Ex"], q["E"][0], q["E"][1]])
    coef = _spline(x, y)
    Ek = [_to_wire(t, _resample(x, y, xw + t.r, coef)) for t, xw in zip(ts, q["wx"])]
    E, H = _dev(q["E"], torch.complex128), _dev(q["H"], torch.complex128)

    def deriv(f):
        return torch.fft.ifft(torch.fft.fft(f) * (1j * qx))
    sg = torch.tensor([[-1.0], [1.0]], dtype=torch.float64, device="cuda")
    H = (H + dt / MU0 * sg * deriv(E)) * mask
    o = _rk4(ts, mats, Ek, [torch.zeros_like(e) for e in Ek], dt)
    Pg, rho = np.zeros((3, nx), complex), np.zeros(nx, complex)
    for t, xw, w in zip(ts, q["wx"], o):
        v = _resample(t.r, w[3].cpu().numpy(), x - xw)
        Pg += v[:3]
        rho += v[4] - v[3]
    J = _dev(Pg[1:] / dt, torch.complex128)
    J[0, q["src"]] += _sheet(q, dx, dt)
    ie = dt / (EPS0 * MAT["epsr"])
    E = (E + ie * sg * deriv(H) - ie * J) * mask
    small = (qx[1] - qx[0]) / 1e4
    rk, pk = (torch.fft.fft(_dev(a, torch.complex128)) for a in (rho, Pg[0]))
    Ex = torch.fft.ifft((-1j * rk - qx * pk) / (EPS0 * MAT["epsr"]) / (qx * qx + small) * qx)
    return dict(P=_packed([w[0] for w in o]), C=_packed([w[1] for w in o]),
                D=_packed([w[2] for w in o]), E=E, H=H, Ex=Ex,
                src=_packed([w[3] for w in o]))


def _curl(F, n, d):
    k = [_dev(_fft_q(m, d)).reshape([-1 if a == c else 1 for c in range(3)]) for a, m in enumerate(n)]
    f = torch.fft.fftn(F, dim=(1, 2, 3))
    return torch.fft.ifftn(torch.stack([1j * (k[1] * f[2] - k[2] * f[1]),
                                        1j * (k[2] * f[0] - k[0] * f[2]),
                                        1j * (k[0] * f[1] - k[1] * f[0])]), dim=(1, 2, 3))


def _mask3(q):
    m = [_dev(_mask(a, b, q["abc"])) for a, b in zip(q["n"], q["n_abc"])]
    return m[0][:, None, None] * m[1][None, :, None] * m[2][None, None, :]


def _exact_field3(case, seed):
    q = _grid3_setup(case, seed)
    g = _gen(seed)
    E, H, dt = q["E"], q["H"], q["dt"]
    E[0] += 1e5 * _cnormal(g, *q["n"])
    J = 1e9 * _cnormal(g, 3, *q["n"])
    mask, ie = _mask3(q), dt / (EPS0 * MAT["epsr"])
    H = (H - dt / MU0 * _curl(E, q["n"], q["d"])) * mask
    E = (E + ie * (_curl(H, q["n"], q["d"]) - J)) * mask
    return dict(E=E, H=H)


def _exact_grid3(case, seed):
    q = _grid3_setup(case, seed)
    ts, mats = _case_tables(case), _wires_inputs(case, seed, coherent=False)
    n, d, dt, E = q["n"], q["d"], q["dt"], q["E"]
    ax = [np.linspace(-(m - 1) * d / 2.0, (m - 1) * d / 2.0, m) for m in n]
    Ek = []
    for t, (xw, yw) in zip(ts, q["xy"]):
        i, fx = _cell(ax[0], xw)
        j, fy = _cell(ax[1], yw)
        ln = ((1 - fx) * (1 - fy) * E[:, i, j] + fx * (1 - fy) * E[:, i + 1, j]
              + (1 - fx) * fy * E[:, i, j + 1] + fx * fy * E[:, i + 1, j + 1])
        Ek.append(_to_wire(t, _resample(ax[2], ln[[2, 0, 1]].cpu().numpy(), t.r)))
    mask, ie = _mask3(q), dt / (EPS0 * MAT["epsr"])
    H = (q["H"] - dt / MU0 * _curl(E, n, d)) * mask
    o = _rk4(ts, mats, Ek, [torch.zeros_like(e) for e in Ek], dt)
    J = torch.zeros_like(E)
    for t, (xw, yw), w in zip(ts, q["xy"], o):
        v = _dev(_resample(t.r, w[3].cpu().numpy(), ax[2])[[1, 2, 0]], torch.complex128)
        gx, gy = (_dev(np.exp(-(a - b) ** 2 / (2.0 * q["gate"] ** 2)))
                  for a, b in ((ax[0], xw), (ax[1], yw)))
        J += (gx[:, None] * gy[None, :])[None, :, :, None] * v[:, None, None, :]
    J /= dt
    beam = np.exp(-(ax[1][:, None] ** 2 + ax[2][None, :] ** 2) / q["waist"] ** 2)
    J[1, q["src"]] += _sheet(q, d, dt) * _dev(beam)
    E = (E + ie * (_curl(H, n, d) - J)) * mask
    return dict(P=_packed([w[0] for w in o]), C=_packed([w[1] for w in o]),
                D=_packed([w[2] for w in o]), E=E, H=H, src=_packed([w[3] for w in o]))


def _cell(g, v):
    i = min(max(int(np.searchsorted(g, v, side="right") - 1), 0), len(g) - 2)
    return i, (v - g[i]) / (g[i + 1] - g[i])


def exact(case, seed):
    return dict(solver=_exact_solver, functions=_exact_functions, rk4=_exact_rk4,
                line=_exact_line, grid3=_exact_grid3, field3=_exact_field3)[case["kind"]](case, seed)
