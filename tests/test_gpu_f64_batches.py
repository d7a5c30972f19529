"""FP64 right-hand side of many wires at once against one of them alone (needs a GPU): the rows of
many small wires are cut into digits several groups to a block, those of a few by pairs of warps.
The two agree within the products' own bound, (2 Nk + 8) 2^-53 of the operands' norms on either
side; general complex states keep the sums from cancelling to less than half of those."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from oracle import sbe_oracle as O  # noqa: E402

MAT = dict(me=0.067 * O.ME0, mh=0.45 * O.ME0, gap=1.52 * O.E0, HO=100e-3 * O.E0, Delta0=6e-9,
           gam_e=1e12, gam_h=1e12, gam_eh=1e12, epsr=12.9, Oph=36e-3 * O.E0 / O.HBAR,
           Gph=3e-3 * O.E0 / O.HBAR)
FLAGS = dict(Optics=True, Excitons=True, EHs=False, Screened=True, Phonon=True, DCTrans=False,
             LF=True, FreePot=False, DiagDph=True, OffDiagDph=True, Recomb=False)


def _rhs(nk, nw):
    from pulsesuite_gb300 import _lib
    from pulsesuite_gb300.wires import WireContext, WireSpec
    ctx = WireContext([WireSpec(nk=nk, L=np.pi / (3e9 / (nk / 2 - 0.5)), temp=300.0,
                                wire_index=1, flags=dict(FLAGS), **MAT) for _ in range(nw)])
    rng = np.random.default_rng(nk)
    z = rng.standard_normal((3, nk, nk)) + 1j * rng.standard_normal((3, nk, nk))
    P, C, D = (ctx.pack([0.05 * m] * nw) for m in z)
    wk = ctx.table(0, "window_k").cpu().numpy()
    Ek = ctx.pack_r([np.stack([0 * wk, 2e7 * wk, 1e7 * wk])] * nw, 3)
    out = [ctx.mat(x, nw - 1).clone() for x in ctx.rhs(P, C, D, Ek, _lib.PREC_FP64)]
    ctx.check()
    ctx.close()
    return out


@pytest.mark.parametrize("nk,nw", ((32, 40), (48, 24), (64, 20), (96, 16), (130, 12), (160, 10),
                                   (288, 3)))
def test_batch_and_single_agree(nk, nw):
    for got, ref in zip(_rhs(nk, nw), _rhs(nk, 1)):
        err = float(torch.linalg.norm(got - ref) / torch.linalg.norm(ref))
        assert err <= 2 * 2 * (2 * nk + 8) * 2.0 ** -53
