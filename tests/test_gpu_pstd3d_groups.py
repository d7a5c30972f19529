"""3-D field transforms of every line length on each axis: FP32 in groups of radix-2 stages, FP64 in
radix 4 (needs a GPU)."""
import math

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from oracle import pstd_oracle as PO  # noqa: E402

LINES = [2, 4, 8, 16, 32, 64, 128, 256, 512, 1024]


def _rel(a, b):
    return float(np.linalg.norm(a.cpu().numpy() - b) / np.linalg.norm(b))


@pytest.mark.parametrize("fp32", [True, False])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("length", LINES)
def test_curl_and_step(axis, length, fp32):
    """Against the oracle.  Tolerance: a stage rounds a sum, a product and a twiddle, each within
    2^-24 of the value in FP32 (3 per stage, forward and inverse), the conversion, the wavenumber
    product and the scaling a few more; in FP64 2^-53, and the oracle's own as much again."""
    from pulsesuite_gb300.pstd import Pstd3D
    n = [4, 8, 2]
    n[axis] = length
    n = tuple(n)
    tol = (6 * math.log2(math.prod(n)) + 8) * (2.0 ** -24 if fp32 else 2.0 ** -52)
    d = (20e-9, 15e-9, 25e-9)
    abc = tuple(min(2, v // 4) for v in n)
    g = Pstd3D(n, d, 12.9, abc, 0.3, fp32_work=fp32)
    o = PO.Pstd3D(n, d, 12.9, abc, 0.3)
    rng = np.random.default_rng(length + axis)
    F, E, H, J = (rng.standard_normal((3,) + n) + 1j * rng.standard_normal((3,) + n)
                  for _ in range(4))
    H *= 0.01
    J *= 1e6
    dev = lambda x: torch.as_tensor(np.ascontiguousarray(x)).cuda()  # noqa: E731
    assert _rel(g.curl(dev(F)), o.curl(F)) < tol
    dt = 1e-17
    Ed, Hd = dev(E), dev(H)
    g.step(Ed, Hd, dev(J), dt)
    Eo, Ho = o.step(E.copy(), H.copy(), J, dt)
    assert _rel(Ed, Eo) < tol and _rel(Hd, Ho) < tol
    g.close()
