"""Small coherences beside large diagonals in the FP64 right-hand side (needs a GPU).

C and D carry the occupations and Hee, Hhh the band energies on their diagonals; the coherences
beside them may be many orders smaller.  Element by element the result stays within what FP64 dot
products of K complex terms allow, (2 K + 8) u sum |a||b| over the element's own products
(u = 2^-53); the reference is formed in extended precision.  Where a row falls off from element to
element (graded) the sums far from the diagonal are smaller than the norms of the rows that meet in
them, and those, without the diagonals of C, D, Hee and Hhh, bound the error instead: 4 u |a||b| for
each of the four products."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

HBAR = 1.0545718176461565e-34
U = 2.0 ** -53


@pytest.mark.parametrize("eps,graded", ((1.0, 0), (1e-4, 0), (1e-8, 0), (1e-14, 0), (1.0, 1), (1e-6, 1)))
@pytest.mark.parametrize("nk", (32, 33, 64, 130))
def test_elements_of_the_derivatives(nk, eps, graded):
    from pulsesuite_gb300 import SBEs
    rng = np.random.default_rng(nk)
    near = np.exp(-20.0 / nk * np.abs(np.arange(nk)[:, None] - np.arange(nk))) if graded else 1.0
    z = lambda: near * (rng.standard_normal((nk, nk)) + 1j * rng.standard_normal((nk, nk)))  # noqa: E731
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
    peeled = [np.abs(np.diag(x)) for x in (C, D, Hee, Hhh)]

    def norms(x, axis):   # of an operand's rows as the products take them
        y = np.abs(x)
        if any(np.array_equal(np.diag(y), d) for d in peeled):
            np.fill_diagonal(y, 0.0)
        return np.linalg.norm(y, axis=axis)
    for f, pairs, extra in cases:
        got = f(*a, *rest).cpu().numpy()
        ref = (sum(wide(x) @ wide(y) for x, y in pairs) + sum(wide(x) for x in extra)) / ih
        S = (sum(np.abs(x) @ np.abs(y) for x, y in pairs) + sum(np.abs(x) for x in extra)) / HBAR
        tol = (2 * nk + 8) * U * S
        if graded:
            tol = tol + 4 * U / HBAR * sum(np.outer(norms(x, 1), norms(y, 0)) for x, y in pairs)
        r = np.abs(got - ref) / tol
        assert np.all(r <= 1), (f.__name__, float(r.max()))
