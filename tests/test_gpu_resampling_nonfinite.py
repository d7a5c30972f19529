"""Prop2QW and QW2Prop of fields with a value that is not finite (needs a GPU): the spline's solve
runs from end to end of the knots, so that part of the field (real or imaginary) is NaN wherever it
is sampled, however far away, and the other fields stay as they are."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from oracle import sbe_oracle as O  # noqa: E402

MAT = dict(me=0.067 * O.ME0, mh=0.45 * O.ME0, gap=1.52 * O.E0, HO=100e-3 * O.E0, Delta0=6e-9,
           gam_e=1e12, gam_h=1e12, gam_eh=1e12, epsr=12.9, Oph=36e-3 * O.E0 / O.HBAR,
           Gph=3e-3 * O.E0 / O.HBAR)


def _context(nk):
    from pulsesuite_gb300.wires import WireContext, WireSpec
    return WireContext([WireSpec(nk=nk, L=np.pi / (3e9 / (nk / 2 - 0.5)), wire_index=1, **MAT)])


@pytest.mark.parametrize("bad", (float("nan"), float("inf")))
@pytest.mark.parametrize("n,at", ((5, 0), (300, 299), (2000, 0), (2000, 1990)))
def test_prop2qw(n, at, bad):
    ctx = _context(64)
    r = ctx.table(0, "r").cpu().numpy()
    rr = np.linspace(10 * r[0], 10 * r[-1], n)
    f = np.stack([np.cos(rr * 1e6 * (i + 1)) + 0.5j for i in range(4)])
    T = lambda x: torch.as_tensor(x).cuda()  # noqa: E731
    ref = ctx.prop2qw(0, T(rr), T(f)).cpu().numpy()
    f[1, at] = complex(bad, 0.5)
    f[2, at] = complex(f[2, at].real, bad)      # the imaginary part is dropped
    got = ctx.prop2qw(0, T(rr), T(f)).cpu().numpy()
    assert np.all(np.isnan(got[1].real)) and np.all(np.isnan(got[1].imag))
    keep = [0, 2, 3]
    assert np.array_equal(got[keep], ref[keep])
    ctx.close()


@pytest.mark.parametrize("nk", (64, 200))
def test_qw2prop(nk):
    ctx = _context(nk)
    r = ctx.table(0, "r").cpu().numpy()
    rr = np.linspace(2 * r[0], 2 * r[-1], 333)
    s = np.stack([np.cos(r * 1e8 * (i + 1)) + 1j * np.sin(r * 1e8) for i in range(5)])
    T = lambda x: torch.as_tensor(x).cuda()  # noqa: E731
    ref = ctx.qw2prop(0, T(rr), T(s), False).cpu().numpy()
    s[3, 2] = complex(s[3, 2].real, float("inf"))
    got = ctx.qw2prop(0, T(rr), T(s), False).cpu().numpy()
    inside = (rr >= r[0]) & (rr <= r[-1])
    assert np.all(np.isnan(got[3].imag[inside])) and np.all(got[3].imag[~inside] == 0)
    assert np.array_equal(got[3].real, ref[3].real)
    keep = [0, 1, 2, 4]
    assert np.array_equal(got[keep], ref[keep])
    ctx.close()
