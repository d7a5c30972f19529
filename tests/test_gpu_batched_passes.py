"""Passes over several buckets in one launch: every wire of a context of many Nk steps to the same
bits as alone (needs a GPU)."""
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


def _state(nk):
    rng = np.random.default_rng(nk)
    z = rng.standard_normal((3, nk, nk)) + 1j * rng.standard_normal((3, nk, nk))
    herm = lambda a: 0.05 * (a + a.conj().T) / np.sqrt(8 * nk)  # noqa: E731
    diag = np.diag(rng.uniform(0, 0.1, nk))
    return 1e-3 * z[0], herm(z[1]) + diag, herm(z[2]) + diag


def _step(nks):
    from pulsesuite_gb300 import _lib
    from pulsesuite_gb300.wires import WireContext, WireSpec
    ctx = WireContext([WireSpec(nk=nk, L=np.pi / (3e9 / (nk / 2 - 0.5)), temp=300.0, wire_index=1,
                                flags=dict(FLAGS), **MAT) for nk in nks])
    st = [_state(nk) for nk in nks]
    P, C, D = (ctx.pack([s[i] for s in st]) for i in range(3))
    wk = [ctx.table(w, "window_k").cpu().numpy() for w in range(len(nks))]
    Ek = ctx.pack_r([np.stack([0 * k, 2e7 * k, 0 * k]) for k in wk], 3)
    src = ctx.zeros_r(5)
    ctx.rk4_step(P, C, D, Ek, torch.zeros_like(Ek), 0.1e-15, src, _lib.PREC_MIXED)
    ctx.check()
    out = [[ctx.mat(x, w).clone() for x in (P, C, D)] + [ctx.rvec(src, w, 5).clone()]
           for w in range(len(nks))]
    ctx.close()
    return out


# one Nk (a common grid), a few (their own grids in one launch), ten (30 parts: two launches)
@pytest.mark.parametrize("nks", [[40, 40, 40], [16, 72, 72, 136],
                                 [8, 16, 24, 32, 40, 48, 64, 72, 96, 128, 128]])
def test_same_bits_as_alone(nks):
    got = _step(nks)
    for w, nk in enumerate(nks):
        for a, b in zip(got[w], _step([nk])[0]):
            assert torch.equal(a, b), nk
