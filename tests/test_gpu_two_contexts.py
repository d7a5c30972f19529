"""Two contexts at work at the same time, each replaying a captured step on a stream of its own
(needs a GPU): each ends with the bits that it reaches alone.  Thousands of launches of the
tensor-core engine overlap those of the other context; those of the larger one have more tiles than
the GPU has SMs, so that its CTAs draw them from the launch's counter.  Between the two captures lie
1011 other launches of the engine: a ring of 1024 counters would give both the same ones."""
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
SIZES = ((256, 6, 1500), (64, 1, 4500))   # Nk, wires, steps: about a second each
LAUNCHES = 13                             # of the engine in one step


class _Run:
    def __init__(self, nk, nw):
        from pulsesuite_gb300 import _lib
        from pulsesuite_gb300.wires import WireContext, WireSpec
        self.prec = _lib.PREC_MIXED
        self.ctx = WireContext([WireSpec(nk=nk, L=np.pi / (3e9 / (nk / 2 - 0.5)), temp=300.0,
                                         wire_index=w + 1, flags=dict(FLAGS), **MAT)
                                for w in range(nw)])
        rng = np.random.default_rng(nk)
        z = rng.standard_normal((3, nk, nk)) + 1j * rng.standard_normal((3, nk, nk))
        herm = [0.02 * (a + a.conj().T) / np.sqrt(8 * nk) + np.diag(rng.uniform(0, 0.1, nk))
                for a in z[1:]]
        self.st = [self.ctx.pack([m] * nw) for m in (1e-3 * z[0], *herm)]
        wk = self.ctx.table(0, "window_k").cpu().numpy()
        self.Ek = self.ctx.pack_r([np.stack([0 * wk, 1e7 * wk, 0 * wk])] * nw, 3)
        self.dEk, self.src = torch.zeros_like(self.Ek), self.ctx.zeros_r(5)
        self.graph = self.ctx.rk4_graph(*self.st, self.Ek, self.dEk, 0.02e-15, self.src, self.prec)
        torch.cuda.synchronize()
        self.stream = torch.cuda.Stream()

    def step(self):
        with torch.cuda.stream(self.stream):
            self.graph.launch()

    def result(self):
        self.stream.synchronize()
        self.ctx.check()
        out = [x.clone() for x in (*self.st, self.src)]
        self.graph.close()
        self.ctx.close()
        return out


def _other_launches(n):
    from pulsesuite_gb300 import _lib
    lib, x = _lib.load(), torch.ones((1, 8, 8), dtype=torch.complex128, device="cuda")
    out = torch.empty_like(x)
    for _ in range(n):
        _lib.check(lib.sbe_tc_selftest(8, 1, _lib.ptr(x), _lib.ptr(x), 0, 0, 1, _lib.ptr(out),
                                       _lib.stream_handle()), "sbe_tc_selftest")


def test_overlapping_contexts_keep_their_bits():
    alone = []
    for nk, nw, steps in SIZES:
        r = _Run(nk, nw)
        for _ in range(steps):
            r.step()
        alone.append(r.result())
    both = [_Run(*SIZES[0][:2])]
    _other_launches(1024 - LAUNCHES)
    both.append(_Run(*SIZES[1][:2]))
    for _ in range(SIZES[0][2]):
        both[0].step()
        for _ in range(SIZES[1][2] // SIZES[0][2]):
            both[1].step()
    for r, ref in zip(both, alone):
        for a, b in zip(r.result(), ref):
            assert bool(torch.isfinite(torch.view_as_real(b)).all()) and torch.equal(a, b)
