"""FP64 contractions on exact-slice tensor-core products (csrc/f64_slices.cu, f64_path.cu)
through the pure functions, at the edges of their 128 x 64 tiles, 32-wide K blocks and
128-deep accumulations, and around Nk = 32 where the SIMT kernels hand over.

Tolerance per element, for each product A B: NumPy's own dot products are within
(2 K + 8) u |A||B| <= (2 K + 8) u |a_row||b_col| (u = 2^-53, complex), the slices within
2^-52 |a_row||b_col| (planes left out and one rounding); dpdt, dCdt, dDdt add four."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

HBAR = 1.0545718176461565e-34
U = 2.0 ** -53
SIZES = (31, 32, 33, 63, 64, 65, 96, 127, 128, 129, 130, 193, 257)


def _inputs(nk, seed=0):
    rng = np.random.default_rng(seed)
    z = lambda: rng.standard_normal((nk, nk)) + 1j * rng.standard_normal((nk, nk))
    # rows of very different size, as occupations that fall off with k make them
    env = np.exp(-8.0 * np.abs(np.linspace(-1, 1, nk)))
    C, D = env[:, None] * z() * env[None, :], env[:, None] * z()
    H = [1e-19 * np.diag(rng.uniform(1, 10, nk)) + 1e-22 * z() for _ in range(2)]
    return C, D, 1e-2 * env[None, :] * z(), 1e-21 * z(), H[0], H[1]


def _bound(pairs, K):
    b = 0.0
    for A, B in pairs:
        b = b + np.linalg.norm(A, axis=1)[:, None] * np.linalg.norm(B, axis=0)[None, :]
    return ((2 * K + 8) * U + 2 * U) * b


@pytest.mark.parametrize("nk", SIZES)
def test_rhs_functions(nk):
    from pulsesuite_gb300 import SBEs
    C, D, p, Heh, Hee, Hhh = _inputs(nk, nk)
    ge, gh = np.full(nk, 1e12), np.full(nk, 2e12)
    off = 1e-25 * p
    T = lambda x: torch.as_tensor(np.ascontiguousarray(x)).cuda()
    a = [T(x) for x in (C, D, p, Heh, Hee, Hhh)]
    rest = (T(ge), T(gh), T(off))
    ih = 1j * HBAR
    cases = (
        (SBEs.dpdt, ((Hhh, p), (-D.T, Heh.T), (p, Hee.T), (-Heh.T, C)),
         Heh.T + off - ih * (ge[None, :] + gh[:, None]) * p),
        (SBEs.dCdt, ((C, Hee.T), (-Hee.T, C), (p.conj().T, Heh.T), (-Heh.conj(), p)), 0.0),
        (SBEs.dDdt, ((D, Hhh.T), (-Hhh.T, D), (p.conj(), Heh), (-Heh.conj().T, p.T)), 0.0))
    for f, pairs, extra in cases:
        got = f(*a, *rest).cpu().numpy()
        ref = (sum(x @ y for x, y in pairs) + extra) / ih
        tol = (_bound(pairs, nk) + 8 * U * np.abs(extra)) / HBAR
        assert np.all(np.abs(got - ref) <= tol), (f.__name__, float(np.max(np.abs(got - ref) / tol)))


@pytest.mark.parametrize("nk", SIZES)
@pytest.mark.parametrize("lf", (True, False))
def test_exchange_sums(nk, lf):
    from oracle import sbe_oracle as O
    from pulsesuite_gb300 import SBEs
    C, D, p, Meh, _, _ = _inputs(nk, nk + 1)
    rng = np.random.default_rng(nk)
    VC = np.zeros((nk, nk, 3))
    VC[:, 0, :] = 1e-21 * rng.uniform(0.1, 1, (nk, 3))
    Ee, Eh, z = rng.uniform(1, 2, nk) * 1e-19, rng.uniform(1, 2, nk) * 1e-20, np.zeros((nk, nk))
    out = [torch.empty((nk, nk), dtype=torch.complex128, device="cuda") for _ in range(3)]
    T = lambda x: torch.as_tensor(np.ascontiguousarray(x)).cuda()
    SBEs.calc_h(T(Meh), T(z), T(z), T(C), T(D), T(p), T(VC), *out, T(Ee), T(Eh), 2e-19, True, lf, False)
    ref = O.calc_h(Meh, z, z, C, D, p, VC, Ee, Eh, 2e-19, True, lf, False)
    # each element: Nk products of |V| <= vmax with the states' diagonals, the direct terms' traces
    # (Nk terms) and the diagonal energies
    vmax, n = VC.max(), np.sqrt(nk)
    for got, r, X in zip(out, ref, (p, C, D)):
        scale = vmax * n * np.linalg.norm(np.abs(C) + np.abs(D) + np.abs(X)) + 1e-18
        assert np.max(np.abs(got.cpu().numpy() - r)) <= (4 * nk + 16) * U * scale


def test_extreme_digits():
    """Every digit below the first at -128: the accumulators reach their bound, and the sum of
    nk equal products is known."""
    from pulsesuite_gb300 import SBEs
    nk = 256                     # the row norm is 16 x: a power of two
    x = float.fromhex("0x1.7f7f7f7f7f7f8p-1")
    one = torch.full((nk, nk), x, dtype=torch.complex128, device="cuda")
    z = torch.zeros_like(one)
    g = torch.zeros(nk, dtype=torch.float64, device="cuda")
    d = SBEs.dpdt(z, z, one, z, z, one, g, g, z)          # Hhh p / (i hbar)
    ref = -1j * (nk * x * x) / HBAR
    assert float((d - ref).abs().max()) <= 4 * U * abs(ref)


@pytest.mark.parametrize("bad", (float("nan"), float("inf")))
def test_non_finite_rows(bad):
    from pulsesuite_gb300 import SBEs
    nk = 96
    C, D, p, Heh, Hee, Hhh = (torch.as_tensor(x).cuda() for x in _inputs(nk, 3))
    ref = SBEs.dDdt(C, D, 0 * p, 0 * Heh, Hee, Hhh, None, None, None)
    D2 = D.clone()
    D2[17, 5] = bad
    got = SBEs.dDdt(C, D2, 0 * p, 0 * Heh, Hee, Hhh, None, None, None)
    # D Hhh^T - Hhh^T D: row 17 of the first product, column 5 of the second
    keep = torch.ones((nk, nk), dtype=torch.bool, device="cuda")
    keep[17, :] = False
    keep[:, 5] = False
    assert bool(torch.isnan(got[17, :].abs()).all()) and bool(torch.isnan(got[:, 5].abs()).all())
    assert bool(torch.isfinite(torch.view_as_real(got)[keep]).all())
    scale = torch.linalg.norm(Hhh) * torch.linalg.norm(D) / HBAR
    assert float((got - ref)[keep].abs().max()) <= 4 * nk * U * float(scale)


@pytest.mark.parametrize("nk,nw", ((4, 1), (6, 2), (32, 3), (34, 5), (64, 8), (66, 9), (130, 1)))
def test_dephasing_sums(nk, nw):
    """De, Dh of groups of one to nine equal wires, k tiles of 32 and chunks of 64 p with
    remainders.  The literal sums round four energies of up to 5.1 eV (k = 3e9 1/m, electrons)
    against hbar gamma = 0.66 meV: 4 u 7750 = 3.5e-12 of a Lorentzian; 1e-11 of the largest."""
    from oracle import sbe_oracle as O
    from pulsesuite_gb300.wires import WireContext, WireSpec
    mat = dict(me=0.067 * O.ME0, mh=0.45 * O.ME0, gap=1.52 * O.E0, HO=100e-3 * O.E0, Delta0=6e-9,
               gam_e=1e12, gam_h=2e12, gam_eh=1.5e12, epsr=12.9, Oph=36e-3 * O.E0 / O.HBAR,
               Gph=3e-3 * O.E0 / O.HBAR)
    L = np.pi / (3e9 / (nk / 2 - 0.5))
    ctx = WireContext([WireSpec(nk=nk, L=L, wire_index=w + 1, **mat) for w in range(nw)])
    rng = np.random.default_rng(nk)
    occ = rng.uniform(0, 0.9, (2, nw, nk))
    C, D = (ctx.pack([np.diag(o).astype(complex) for o in occ[s]]) for s in range(2))
    De, Dh = (x.cpu().numpy().reshape(nw, 2 * nk + 1, nk) for x in ctx.deph(C, D))
    E = O.wire_constants(mat, O.wire_grid(nk, L)["kr"])
    for w in range(nw):
        ne, nh = (torch.as_tensor(occ[s][w].astype(complex)).cuda() for s in range(2))
        VC = ctx.screened_arrays(w, ne, nh)[0].cpu().numpy()
        for got, ref in ((De[w], O.offdiag_De(occ[0][w], occ[1][w], E["Ee"], E["Eh"], mat["gam_eh"],
                                              mat["gam_h"], VC)),
                         (Dh[w], O.offdiag_Dh(occ[0][w], occ[1][w], E["Ee"], E["Eh"], mat["gam_e"],
                                              mat["gam_h"], VC))):
            assert np.max(np.abs(got - ref)) <= 1e-11 * np.max(np.abs(ref))
    ctx.close()
