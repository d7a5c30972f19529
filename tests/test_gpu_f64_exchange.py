"""Exchange sums of the FP64 Hamiltonians element by element (the comparison with the GPU needs one).

Element (a, b) of the sums is a product of row a of the Toeplitz operand V and the diagonal b - a of
the state, so its error is measured by their two norms: 4 u for the digit planes and their rounding
(u = 2^-53), 8 u of the element and of what else is added to it, and (Nk / 16 + 16) u of the
magnitudes in the traces of the direct terms; the energies count on the diagonal alone.  The
reference is formed in extended precision.  Operands of 44 bits fail this by far."""
import numpy as np
import pytest

U = 2.0 ** -53
SIZES = (32, 33, 64, 65, 128, 129)


def _inputs(nk, graded):
    rng = np.random.default_rng(nk)
    z = lambda: rng.standard_normal((nk, nk)) + 1j * rng.standard_normal((nk, nk))  # noqa: E731
    env = np.exp(-6.0 * np.abs(np.linspace(-1, 1, nk))) if graded else np.ones(nk)
    C, D, p = (s * env[:, None] * z() * env[None, :] for s in (1.0, 0.5, 1e-2))
    VC = np.zeros((nk, nk, 3))
    VC[:, 0, :] = 1e-21 * (rng.uniform(0.5, 1, (nk, 3)) / (1.0 + np.arange(nk)[:, None]))
    return p, C, D, 1e-22 * z(), VC, rng.uniform(1, 2, nk) * 1e-19, rng.uniform(1, 2, nk) * 1e-20


def _toeplitz(v):
    nk = len(v)
    q = np.abs(np.arange(nk)[:, None] - np.arange(nk)[None, :])
    T = v[q]
    np.fill_diagonal(T, 0.0)
    return T


def _exchange(v, X, cut=None):
    """sum_t V(|t - a|) X[t + b - a][t] and the norms |V row a| |diagonal b - a of X|; cut: the
    operands rounded to so many bits of their norms."""
    nk = len(v)
    T = _toeplitz(v)
    B = np.zeros((nk, 2 * nk - 1), complex)
    for d in range(-(nk - 1), nk):
        t = np.arange(max(0, -d), min(nk, nk - d))
        B[t, d + nk - 1] = X[t + d, t]
    nT, nB = np.linalg.norm(T, axis=1), np.linalg.norm(B, axis=0)
    if cut:
        r = lambda x, n: np.rint(x / n * 2.0 ** cut) * n * 2.0 ** -cut  # noqa: E731
        T = r(T, nT[:, None])
        n = np.where(nB > 0, nB, 1.0)
        B = r(B.real, n) + 1j * r(B.imag, n)
    Tw = T.astype(np.longdouble)
    S = Tw @ B.real.astype(np.longdouble) + 1j * (Tw @ B.imag.astype(np.longdouble))
    a, b = np.mgrid[:nk, :nk]
    return S[a, b - a + nk - 1], (nT[:, None] * nB[None, :])[a, b - a + nk - 1]


def _reference(p, C, D, Meh, VC, Ee, Eh, gap, cut=None):
    """Heh, Hee, Hhh (SBEs.py:1044-1131 with excitons and LF) and the bound of each element."""
    nk = len(Ee)
    a, b = np.mgrid[:nk, :nk]
    d = np.abs(a - b)
    out = []
    for n, X in enumerate((p, C, D)):
        x, s = _exchange(VC[:, 0, n], X, cut)
        H = (Meh if n == 0 else np.diag((Ee + gap, Eh)[n - 1])).astype(np.clongdouble)
        tol = 4 * s + 8 * (np.abs(H) + np.abs(x))
        if n == 0:
            H = H + x
        else:
            tr = [np.array([np.trace(Y.astype(np.clongdouble), offset=o) for o in range(-nk + 1, nk)])
                  for Y in (X, (D, C)[n - 1])]
            mag = [np.array([np.trace(np.abs(Y), offset=o) for o in range(-nk + 1, nk)])
                   for Y in (X, (D, C)[n - 1])]
            v, v0 = VC[:, 0, n][d], VC[:, 0, 0][d]
            o = a - b + nk - 1
            direct = v * tr[0][o] - v0 * tr[1][2 * (nk - 1) - o]
            off = a != b
            H = H - x + np.where(off, direct, 0)
            tol = tol + np.where(off, (nk / 16 + 16) * (v * mag[0][o] + v0 * mag[1][2 * (nk - 1) - o]), 0)
        out.append((H, U * tol))
    return out


@pytest.mark.parametrize("nk", SIZES)
def test_bound_sees_44_bits(nk):
    args = _inputs(nk, False)
    for (ref, tol), (cut, _) in zip(_reference(*args, 2e-19), _reference(*args, 2e-19, cut=44)):
        off = ~np.eye(nk, dtype=bool)
        assert np.max((np.abs(cut - ref) / tol)[off]) > 2


@pytest.mark.gpu
@pytest.mark.parametrize("graded", (False, True))
@pytest.mark.parametrize("nk", SIZES)
def test_elements_of_the_hamiltonians(nk, graded):
    torch = pytest.importorskip("torch")
    from pulsesuite_gb300 import SBEs
    p, C, D, Meh, VC, Ee, Eh = args = _inputs(nk, graded)
    T = lambda x: torch.as_tensor(np.ascontiguousarray(x)).cuda()  # noqa: E731
    z = T(np.zeros((nk, nk), complex))
    out = [torch.empty((nk, nk), dtype=torch.complex128, device="cuda") for _ in range(3)]
    SBEs.calc_h(T(Meh), z, z, T(C), T(D), T(p), T(VC), *out, T(Ee), T(Eh), 2e-19, True, True, False)
    for got, (ref, tol) in zip(out, _reference(*args, 2e-19)):
        r = np.abs(got.cpu().numpy() - ref) / tol
        assert np.all(r <= 1), float(r.max())
