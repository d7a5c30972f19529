"""Resampling splines (csrc/spline.cu) through prop2qw and qw2prop against the serial solve: knots
on both sides of the 64-point tiles, the 8-point segments and the warm-up ranges, uniform and
graded spacings (adjacent ratios up to 20).

Tolerance: both solves are backward stable tridiagonal eliminations of a diagonally dominant
system; the warm-ups add 2^-56 at most, the reciprocals an ulp each: 64 u of the largest value."""
import numpy as np
import pytest
import torch

from oracle import sbe_oracle as O

pytestmark = pytest.mark.gpu
TOL = 64 * 2.0 ** -53


def _ctx(nk=16):
    from pulsesuite_gb300.wires import WireContext, WireSpec
    return WireContext([WireSpec(nk=nk, L=50e-9)])


@pytest.mark.parametrize("n", (2, 3, 4, 5, 8, 9, 63, 64, 65, 66, 100, 101, 102, 127, 129, 165, 166,
                               192, 193, 229, 230, 257, 1000))
@pytest.mark.parametrize("grid", ("uniform", "graded", "steep"))
def test_prop2qw_grids(n, grid):
    ctx = _ctx()
    rng = np.random.default_rng(n)
    if grid == "uniform":
        rr = np.linspace(-60e-9, 60e-9, n)
    else:
        # steep: spacings over eight decades (the pivots' own recurrence)
        d = 10.0 ** (rng.uniform(-0.65, 0.65, n - 1) * (1.0 if grid == "graded" else 6.0))
        rr = np.concatenate([[0.0], np.cumsum(d)])
        rr = -60e-9 + 120e-9 * rr / rr[-1]
    f = rng.standard_normal((4, n)) + 1j * rng.standard_normal((4, n))
    got = ctx.prop2qw(0, torch.as_tensor(rr).cuda(), torch.as_tensor(f).cuda()).cpu().numpy()
    r, win = ctx.table(0, "r").cpu().numpy(), ctx.table(0, "window").cpu().numpy()
    ref = np.stack(O.prop2qw(rr, *f, r, win))
    vals = max(np.max(np.abs(O.rescale_1d(rr, a, r) * win)) for a in f)
    assert np.max(np.abs(got - ref)) <= TOL * max(vals, 1.0)
    ctx.close()


@pytest.mark.parametrize("nk", (4, 14, 31, 32, 48, 114))
def test_qw2prop_wires(nk):
    ctx = _ctx(nk)
    rng = np.random.default_rng(nk)
    nr = 2 * nk + 2
    rr = np.linspace(-70e-9, 70e-9, 333)
    s = rng.standard_normal((5, nr)) + 1j * rng.standard_normal((5, nr))
    r = ctx.table(0, "r").cpu().numpy()
    for plas in (False, True):
        got = ctx.qw2prop(0, torch.as_tensor(rr).cuda(), torch.as_tensor(s).cuda(), plas).cpu().numpy()
        ref = np.stack(O.qw2prop(r, *[O.fftg(a) for a in s], rr, plas))
        # the reference's FFT round trip adds log2(Nr) u
        assert np.max(np.abs(got - ref)) <= 2 * TOL * np.max(np.abs(ref))
    ctx.close()
