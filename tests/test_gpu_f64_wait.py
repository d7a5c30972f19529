"""A bounded wait of the FP64 products that gives up: the tiles are NaN, the context it belongs to
reports it, and no other (needs a GPU; each self-test waits about 2 s for operands that never
arrive)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from oracle import sbe_oracle as O  # noqa: E402

MAT = dict(me=0.067 * O.ME0, mh=0.45 * O.ME0, gap=1.52 * O.E0, HO=100e-3 * O.E0, Delta0=6e-9,
           gam_e=1e12, gam_h=1e12, gam_eh=1e12, epsr=12.9, Oph=36e-3 * O.E0 / O.HBAR,
           Gph=3e-3 * O.E0 / O.HBAR)


def _context():
    from pulsesuite_gb300.wires import WireContext, WireSpec
    return WireContext([WireSpec(nk=64, L=np.pi / (3e9 / 31.5), wire_index=1, **MAT)])


def test_flag_of_its_own_context():
    from pulsesuite_gb300 import _lib
    a, b = _context(), _context()
    flags = a.wait_flag(), b.wait_flag()
    tile = a.f64_wait_selftest()
    b.check()                                   # the failure is not b's
    assert [f.value != 0 for f in flags] == [True, False]
    with pytest.raises(_lib.SbeError):
        a.check()
    a.check()                                   # reported once
    assert flags[0].value == 0
    assert bool(torch.isnan(tile).all())
    z = torch.ones((64, 64), dtype=torch.complex128, device="cuda")
    from pulsesuite_gb300 import SBEs
    g = torch.zeros(64, dtype=torch.float64, device="cuda")
    assert bool(torch.isfinite(torch.view_as_real(SBEs.dpdt(z, z, z, z, z, z, g, g, z))).all())
    a.close()
    b.close()


@pytest.mark.parametrize("batch", (False, True))
def test_solver_raises(batch):
    from pulsesuite_gb300 import SBEs, _lib
    rr = np.linspace(-1e-7, 1e-7, 300)
    params = dict(MAT, L=80e-9, Edc=0.0, jmax=1000, ntmax=100)
    flags = dict(Optics=True, Excitons=True, EHs=False, Screened=True, Phonon=True, DCTrans=False,
                 LF=True, FreePot=False, DiagDph=True, OffDiagDph=True, Recomb=False)
    sv = SBEs.SBESolver(None, rr, 0.0, 2e7, 8e-7, 1, True, params=params, flags=flags, batch=batch)
    sv.write_info = False
    f = [2e7 * np.exp(-(rr / 5e-8) ** 2).astype(complex)] * 3 + [np.zeros(300, complex)]
    o = [np.zeros(300, complex) for _ in range(4)]
    step = lambda: sv.QWCalculator(*f, rr, None, 0.05e-15, 1, *o, [False], [False])  # noqa: E731
    step()
    sv.contexts[0].f64_wait_selftest()
    with pytest.raises(_lib.SbeError):
        step()
    step()
    assert np.all(np.isfinite(o[0])) and np.any(o[0] != 0)
