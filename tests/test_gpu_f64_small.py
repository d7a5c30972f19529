"""Small coherences beside large diagonals in the FP64 right-hand side (needs a GPU).

C and D carry the occupations and Hee, Hhh the band energies on their diagonals; the coherences
beside them may be many orders smaller.  Element by element the result stays within what FP64 dot
products of K complex terms allow, (2 K + 8) u sum |a||b| over the element's own products
(u = 2^-53); the reference is formed in extended precision."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

HBAR = 1.0545718176461565e-34
U = 2.0 ** -53


@pytest.mark.parametrize("eps", (1.0, 1e-4, 1e-8, 1e-14))
@pytest.mark.parametrize("nk", (32, 33, 64, 130))
def test_elements_of_the_derivatives(nk, eps):
    from pulsesuite_gb300 import SBEs
    rng = np.random.default_rng(nk)
    z = lambda: rng.standard_normal((nk, nk)) + 1j * rng.standard_normal((nk, nk))  # noqa: E731
    C, D = (eps * 1e-2 * z() for _ in range(2))
    Hee, Hhh = (eps * 1e-22 * z() for _ in range(2))
    for X, lo, hi in ((C, 0.05, 0.1), (D, 0.05, 0.1), (Hee, 2e-19, 3e-19), (Hhh, 1e-20, 1e-19)):
        np.fill_diagonal(X, rng.uniform(lo, hi, nk))
    p, Heh = 1e-2 * eps * z(), 1e-21 * eps * z()
    ge, gh = np.full(nk, 1e12), np.full(nk, 2e12)
    off = 1e-25 * p
    T = lambda x: torch.as_tensor(np.ascontiguousarray(x)).cuda()  # noqa: E731
    a = [T(x) for x in (C, D, p, Heh, Hee, Hhh)]
    rest = (T(ge), T(gh), T(off))
    ih = 1j * HBAR
    cases = (
        (SBEs.dpdt, ((Hhh, p), (-D.T, Heh.T), (p, Hee.T), (-Heh.T, C)),
         (Heh.T, off, -ih * (ge[None, :] + gh[:, None]) * p)),
        (SBEs.dCdt, ((C, Hee.T), (-Hee.T, C), (p.conj().T, Heh.T), (-Heh.conj(), p)), ()),
        (SBEs.dDdt, ((D, Hhh.T), (-Hhh.T, D), (p.conj(), Heh), (-Heh.conj().T, p.T)), ()))
    wide = lambda x: x.astype(np.clongdouble)  # noqa: E731
    for f, pairs, extra in cases:
        got = f(*a, *rest).cpu().numpy()
        ref = (sum(wide(x) @ wide(y) for x, y in pairs) + sum(wide(x) for x in extra)) / ih
        S = (sum(np.abs(x) @ np.abs(y) for x, y in pairs) + sum(np.abs(x) for x in extra)) / HBAR
        r = np.abs(got - ref) / ((2 * nk + 8) * U * S)
        assert np.all(r <= 1), (f.__name__, float(r.max()))
