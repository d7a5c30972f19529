"""The first FP64 step of a context while a graph is being captured elsewhere (needs a GPU): the step
takes the products that it takes otherwise, to the same bits, and the capture stays valid."""
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from oracle import sbe_oracle as O  # noqa: E402

MAT = dict(me=0.067 * O.ME0, mh=0.45 * O.ME0, gap=1.52 * O.E0, HO=100e-3 * O.E0, Delta0=6e-9,
           gam_e=1e12, gam_h=1e12, gam_eh=1e12, epsr=12.9, Oph=36e-3 * O.E0 / O.HBAR,
           Gph=3e-3 * O.E0 / O.HBAR)


def _setup(nk=64):
    from pulsesuite_gb300 import _lib
    from pulsesuite_gb300.wires import WireContext, WireSpec
    ctx = WireContext([WireSpec(nk=nk, L=np.pi / (3e9 / (nk / 2 - 0.5)), wire_index=1, **MAT)])
    rng = np.random.default_rng(nk)
    z = rng.standard_normal((3, nk, nk)) + 1j * rng.standard_normal((3, nk, nk))
    st = [ctx.pack([1e-2 * m]) for m in z]
    wk = ctx.table(0, "window_k").cpu().numpy()
    Ek = ctx.pack_r([np.stack([0 * wk, 2e7 * wk, 0 * wk])], 3)
    dEk, src = torch.zeros_like(Ek), ctx.zeros_r(5)
    return ctx, st, lambda: ctx.rk4_step(*st, Ek, dEk, 0.1e-15, src, _lib.PREC_FP64)


@pytest.mark.parametrize("thread", (False, True))
def test_first_step_beside_a_capture(thread):
    ctx, ref, step = _setup()
    step()
    ctx.check()
    ctx.close()
    ctx, st, step = _setup()
    x = torch.zeros(1000, device="cuda")
    x.add_(1.0)
    graph, other = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()

    def first():
        with torch.cuda.stream(other):
            step()
    with torch.cuda.graph(graph):
        x.add_(1.0)
        if thread:
            t = threading.Thread(target=first)
            t.start()
            t.join()
        else:
            first()
        x.add_(1.0)
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert float(x[0]) == 3.0
    ctx.check()
    for a, b in zip(st, ref):
        assert torch.equal(a, b)
    ctx.close()
