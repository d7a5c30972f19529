"""N tiles of the tensor-core engine: a launch with few tiles takes narrower ones, and the width
changes no bit of a wire's step (needs a GPU)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from oracle import sbe_oracle as O  # noqa: E402

MAT = dict(me=0.067 * O.ME0, mh=0.45 * O.ME0, gap=1.52 * O.E0, HO=100e-3 * O.E0, Delta0=6e-9,
           gam_e=1e12, gam_h=1e12, gam_eh=1e12, epsr=12.9, Oph=36e-3 * O.E0 / O.HBAR,
           Gph=3e-3 * O.E0 / O.HBAR)
# no off-diagonal dephasing: its sums are grouped by the number of wires
FLAGS = dict(Optics=True, Excitons=True, EHs=False, Screened=True, Phonon=True, DCTrans=False,
             LF=True, FreePot=False, DiagDph=True, OffDiagDph=False, Recomb=False)


def _step(nk, nw):
    from pulsesuite_gb300 import _lib
    from pulsesuite_gb300.wires import WireContext, WireSpec
    ctx = WireContext([WireSpec(nk=nk, L=np.pi / (3e9 / (nk / 2 - 0.5)), temp=300.0,
                                wire_index=1, flags=dict(FLAGS), **MAT) for _ in range(nw)])
    rng = np.random.default_rng(nk)
    z = rng.standard_normal((3, nk, nk)) + 1j * rng.standard_normal((3, nk, nk))
    herm = lambda a: 0.05 * (a + a.conj().T) / np.sqrt(8 * nk)  # noqa: E731
    diag = np.diag(rng.uniform(0, 0.1, nk))
    one = [1e-3 * z[0], herm(z[1]) + diag, herm(z[2]) + diag]
    P, C, D = (ctx.pack([m] * nw) for m in one)
    wk = ctx.table(0, "window_k").cpu().numpy()
    Ek = ctx.pack_r([np.stack([0 * wk, 2e7 * wk, 0 * wk])] * nw, 3)
    dEk = torch.zeros_like(Ek)
    src = ctx.zeros_r(5)
    ctx.rk4_step(P, C, D, Ek, dEk, 0.1e-15, src, _lib.PREC_MIXED)
    ctx.check()
    out = [ctx.mat(x, nw - 1).clone() for x in (P, C, D)]
    out.append(ctx.rvec(src, nw - 1, 5).clone())
    ctx.close()
    return out


# the tile edges and the last tile's remainders; 1 wire is narrow in every launch, 3 in some,
# 48 (16 from 256 up) in none
@pytest.mark.parametrize("nk", [8, 32, 56, 64, 72, 128, 136, 192, 256, 264, 320])
def test_width_changes_no_bit(nk):
    many = 48 if nk < 256 else 16
    ref = _step(nk, many)
    assert all(bool(torch.isfinite(torch.view_as_real(r)).all()) for r in ref)
    for nw in (1, 3):
        for a, b in zip(_step(nk, nw), ref):
            assert torch.equal(a, b)
