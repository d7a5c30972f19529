"""Host staging of the drop-in solver's fields (needs a GPU)."""
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


def _solver(n, nw=1, batch=False):
    from pulsesuite_gb300 import SBEs
    rr = np.linspace(-1e-7, 1e-7, n)
    params = dict(MAT, L=40e-9, Edc=0.0, jmax=1000, ntmax=100)
    sv = SBEs.SBESolver(None, rr, 0.0, 2e7, 8e-7, nw, True, params=params, flags=dict(FLAGS),
                        batch=batch)
    sv.write_info = False
    return sv, rr


def _fields(rr, a):
    g = np.exp(-(rr / 5e-8) ** 2)
    return [a * g.astype(complex), 0.5 * a * g + 0j, 0.1 * a * g + 0j, np.zeros(len(rr), complex)]


def _call(sv, rr, f, w=1):
    o = [np.zeros(len(rr), complex) for _ in range(4)]
    sv.QWCalculator(*f, rr, None, 0.05e-15, w, *o, [False], [False])
    return o


def test_wire_staged_again_before_the_last_one():
    """A driver that starts again at wire 1 while that wire's transfer is still under way: the
    first call's field reaches the device whole."""
    n = 200000
    sv, rr = _solver(n, nw=2, batch=True)
    first, second = _fields(rr, 2e7), _fields(rr, -3e7)
    _call(sv, rr, second)                      # buffers
    torch.cuda.synchronize()
    got = []
    busy = torch.empty(1 << 28, dtype=torch.float32, device="cuda")
    for _ in range(5):
        for _ in range(20):
            busy.mul_(1.0)                     # keeps the transfer waiting in the stream
        RR, f4 = sv._stage(1, rr, first)
        got.append(f4.clone())
        sv._stage(1, rr, second)
    ref = torch.as_tensor(np.stack(first))
    for g in got:
        assert torch.equal(g.cpu(), ref)


def test_pinned_memory_refused(monkeypatch):
    """Without pinned memory the solver copies from pageable memory, with the same results."""
    sv, rr = _solver(300)
    f = _fields(rr, 2e7)
    ref = [x.copy() for x in _call(sv, rr, f)]

    def refuse(self, *a, **k):
        raise RuntimeError("CUDA error: out of memory")
    sv, rr = _solver(300)
    monkeypatch.setattr(torch.Tensor, "pin_memory", refuse)
    for a, b in zip(_call(sv, rr, f), ref):
        assert np.array_equal(a, b)



def test_field_shapes():
    """Fields of shapes of their own are refused, as np.stack refuses them; column vectors and
    lists serve."""
    sv, rr = _solver(300)
    f = _fields(rr, 2e7)
    ref = _call(sv, rr, f)
    for bad in (np.zeros(1, complex), np.zeros(299, complex), 0.0):
        sv, rr = _solver(300)
        with pytest.raises(ValueError):
            _call(sv, rr, f[:3] + [bad])
    sv, rr = _solver(300)
    for a, b in zip(_call(sv, rr, [x[:, None] for x in f]), ref):
        assert np.array_equal(a, b)
    sv, rr = _solver(300)
    for a, b in zip(_call(sv, list(rr), f[:3] + [list(f[3])]), ref):
        assert np.array_equal(a, b)
