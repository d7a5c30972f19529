"""1-D field transforms with every number of lines per block (needs a GPU).  FP64: each of the
2 log2 n radix-2 stages rounds a sum, a product and a twiddle, 3 x 2^-53 apiece, and NumPy's the
same: (12 log2 n + 8) 2^-53 stays below the 1e-13 of the other transform tests."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from oracle import pstd_oracle as PO  # noqa: E402

EPSR = 12.9


def _rel(a, b):
    return float(np.linalg.norm(a.cpu().numpy() - b) / np.linalg.norm(b))


@pytest.mark.parametrize("nx", [1 << k for k in range(8, 17)])
def test_derivative_and_longitudinal_field(nx):
    from pulsesuite_gb300.pstd import Pstd1D
    tol = (12 * np.log2(nx) + 8) * 2.0 ** -53
    p = Pstd1D(nx, 10e-9, EPSR)
    _, q = PO.pstd_grid(nx, 10e-9)
    rng = np.random.default_rng(nx)
    f = rng.standard_normal((3, nx)) + 1j * rng.standard_normal((3, nx))
    dev = lambda x: torch.as_tensor(np.ascontiguousarray(x)).cuda()  # noqa: E731
    two = p.deriv(dev(f[:2]))
    for c in range(2):
        assert _rel(two[c], PO.deriv(f[c], q)) < tol
    assert _rel(p.deriv(dev(f[2])), PO.deriv(f[2], q)) < tol
    assert _rel(p.elong(dev(f[0]), dev(1e-9 * f[1])), PO.elong(f[0], 1e-9 * f[1], q, EPSR)) < tol
    p.close()
