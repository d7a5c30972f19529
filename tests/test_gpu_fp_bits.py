"""The FP64 reciprocal and quotient of csrc/fp_bits.cuh against CUDA's division and against extended
precision (needs a GPU and nvcc)."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

PROGRAM = """
#include "fp_bits.cuh"
__global__ void k(long long n, const double* x, const double* d, double* rc, double* own, double* q,
                  double* div) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  rc[i] = sbe::rcp64(x[i]);
  own[i] = 1.0 / x[i];
  const double r = 1.0 / d[i];
  q[i] = sbe::div_by(x[i], d[i], r);
  div[i] = x[i] / d[i];
}
extern "C" int run(long long n, const double* x, const double* d, double* rc, double* own, double* q,
                   double* div) {
  k<<<(unsigned)((n + 255) / 256), 256>>>(n, x, d, rc, own, q, div);
  return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    from pulsesuite_gb300 import build
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    tmp = tmp_path_factory.mktemp("fp_bits")
    (tmp / "fp.cu").write_text(PROGRAM)
    csrc = Path(build.CSRC)
    subprocess.run([build.nvcc(), "-shared", "-Xcompiler", "-fPIC", "-std=c++17", *build.ARCH, "-I",
                    str(csrc), str(tmp / "fp.cu"), "-o", str(tmp / "fp.so")], check=True)
    lib = ctypes.CDLL(str(tmp / "fp.so"))

    def call(x, d):
        t = [torch.as_tensor(np.ascontiguousarray(a)).cuda() for a in (x, d)]
        o = [torch.empty_like(t[0]) for _ in range(4)]
        torch.cuda.synchronize()
        assert lib.run(ctypes.c_longlong(len(x)), *[ctypes.c_void_p(a.data_ptr()) for a in t + o]) == 0
        return [a.cpu().numpy() for a in o]
    return call


def _random(n, lo, hi, seed):
    rng = np.random.default_rng(seed)
    m = 1.0 + rng.integers(0, 1 << 52, n) * 2.0 ** -52
    m[:64] = 1.0 + np.arange(64) * 2.0 ** -52             # and the ends of the mantissa's range
    m[64:128] = 2.0 - (1 + np.arange(64)) * 2.0 ** -52
    return np.ldexp(m * rng.choice((-1.0, 1.0), n), rng.integers(lo, hi, n))


@pytest.mark.parametrize("lo,hi", ((-3, 3), (-160, -120), (-1021, 1021)))
def test_reciprocal(run, lo, hi):
    x = _random(1 << 18, lo, hi, 1)
    rc, own, _, _ = run(x, x)
    err = np.abs(rc.astype(np.longdouble) - np.longdouble(1) / x.astype(np.longdouble))
    assert np.max(err / np.spacing(np.abs(own))) <= 0.6
    assert np.max(np.abs(rc - own) / np.spacing(np.abs(own))) <= 1


def test_reciprocal_outside_its_range(run):
    x = np.array([0.0, -0.0, 5e-324, -1e-310, np.inf, -np.inf, np.nan])
    assert np.all(np.isnan(run(x, np.ones_like(x))[0]))


@pytest.mark.parametrize("lo,hi", ((-3, 3), (-60, 40), (-900, 900)))
def test_quotient(run, lo, hi):
    n = 1 << 18
    x, d = _random(n, lo, hi, 2), _random(n, max(lo, -60), min(hi, 60), 3)
    d[:4] = 20.0, 0.05e-15, 2e-17, 0.1
    _, _, q, div = run(x, d)
    assert np.array_equal(q, div)


def test_quotient_at_the_ends(run):
    x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e308, 1e-300, 3e-310, 5e-324])
    for d in (0.05e-15, 20.0):
        _, _, q, div = run(x, np.full_like(x, d))
        fin = np.isfinite(div)
        assert np.array_equal(q[~fin], div[~fin], equal_nan=True)
        assert np.all(np.abs(q[fin] - div[fin]) <= np.spacing(np.abs(div[fin])))
