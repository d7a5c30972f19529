"""Coulomb tables of wires listed in any order of their Nk: the same as of each wire alone (needs a
GPU).  The tables are laid out by Nk, the wires come as listed."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from oracle import sbe_oracle as O  # noqa: E402

MAT = dict(me=0.067 * O.ME0, mh=0.45 * O.ME0, gap=1.52 * O.E0, HO=100e-3 * O.E0, Delta0=6e-9,
           gam_e=1e12, gam_h=1e12, gam_eh=1e12, epsr=12.9, Oph=36e-3 * O.E0 / O.HBAR,
           Gph=3e-3 * O.E0 / O.HBAR)


def _tables(nks):
    from pulsesuite_gb300.wires import WireContext, WireSpec
    ctx = WireContext([WireSpec(nk=nk, L=np.pi / (3e9 / (nk / 2 - 0.5)), temp=300.0,
                                wire_index=1, **MAT) for nk in nks])
    out = [ctx.table(w, "V0").clone() for w in range(len(nks))]
    ctx.close()
    return out


@pytest.mark.parametrize("nks", [[96, 40, 64], [64, 8, 128, 8, 32, 200], [200, 128, 64, 32, 8]])
def test_tables_in_any_order(nks):
    for nk, got in zip(nks, _tables(nks)):
        assert torch.equal(got, _tables([nk])[0]), nk
