"""FP32 dephasing sums of several groups of wires in one launch (needs a GPU): each wire's are the
bits that its group reaches in a context of its own, whatever Nk the others have.  Groups of less
than 4 wires, of up to 8 and of up to 16 take kernels of their own."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from oracle import sbe_oracle as O  # noqa: E402

MAT = dict(me=0.067 * O.ME0, mh=0.45 * O.ME0, gap=1.52 * O.E0, HO=100e-3 * O.E0, Delta0=6e-9,
           gam_e=1e12, gam_h=1e12, gam_eh=1e12, epsr=12.9, Oph=36e-3 * O.E0 / O.HBAR,
           Gph=3e-3 * O.E0 / O.HBAR)


def _sums(nks):
    """De, Dh of every wire of a context, the occupations those of its Nk."""
    from pulsesuite_gb300.wires import WireContext, WireSpec
    ctx = WireContext([WireSpec(nk=nk, L=np.pi / (3e9 / (nk / 2 - 0.5)), temp=300.0, wire_index=1,
                                **MAT) for nk in nks])
    occ = [np.random.default_rng(nk).uniform(0, 0.5, (2, nk)) for nk in nks]
    C, D = (ctx.pack([np.diag(o[s]).astype(complex) for o in occ]) for s in range(2))
    De, Dh = ctx.deph(C, D, fp32=True)
    torch.cuda.synchronize()
    # the packed layout: by ascending Nk, the caller's order within one
    out, at = [None] * len(nks), 0
    for w in sorted(range(len(nks)), key=lambda w: nks[w]):
        n = (2 * nks[w] + 1) * nks[w]
        out[w] = [x.reshape(-1)[at:at + n].clone() for x in (De, Dh)]
        at += n
    ctx.close()
    return out


# the second has a wire that takes the per-wire kernel beside a group whose Nk that kernel has no
# shared memory for
@pytest.mark.parametrize("groups", (((64, 1), (136, 5), (72, 12), (40, 3), (520, 1)),
                                    ((64, 1), (1544, 4))))
def test_same_bits_as_alone(groups):
    got = _sums([nk for nk, n in groups for _ in range(n)])
    w = 0
    for nk, n in groups:
        for ref in _sums([nk] * n):
            for a, b in zip(got[w], ref):
                assert bool(a.abs().max() > 0) and torch.equal(a, b), nk
            w += 1
