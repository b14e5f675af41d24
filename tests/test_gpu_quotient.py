"""quotient32 (csrc/quotient.cuh), the one rounding of a cell's centre of mass that is
not a plain FP64 division, against (float)(s / m) in NumPy: quotients on and beside
the middle of two floats and on powers of two, zeros, the smallest and the largest
magnitudes, infinities and NaN.  Compared bit for bit.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = r"""
#include "quotient.cuh"
__global__ void k(const double *s, const double *m, const float *f, float *q, double *w, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        q[i] = nbx::quotient32(s[i], m[i]);
        w[i] = nbx::widen(f[i]);
    }
}
extern "C" int run(const double *s, const double *m, const float *f, float *q, double *w, int n) {
    k<<<(n + 255) / 256, 256>>>(s, m, f, q, w, n);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def run(cuda, tmp_path_factory):
    import torch
    from nns_gb300 import build as nb
    d = tmp_path_factory.mktemp("quotient")
    src, so = str(d / "q.cu"), str(d / "q.so")
    open(src, "w").write(SOURCE)
    subprocess.run([nb.nvcc()] + nb.ARCH + ["-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I",
                                            os.path.join(ROOT, "nns_gb300", "csrc"), src, "-o", so], check=True)
    fn = C.CDLL(so).run

    def call(s, m, f):
        n = len(s)
        dev = [torch.as_tensor(a, device="cuda") for a in (s, m, f)]
        q = torch.empty(n, dtype=torch.float32, device="cuda")
        w = torch.empty(n, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        assert fn(*[C.c_void_p(t.data_ptr()) for t in (*dev, q, w)], n) == 0
        return q.cpu().numpy(), w.cpu().numpy()
    return call


def _same(a, b):
    return np.array_equal(np.isnan(a), np.isnan(b)) and np.array_equal(
        a[~np.isnan(a)].view(np.uint32 if a.dtype == np.float32 else np.uint64),
        b[~np.isnan(b)].view(np.uint32 if b.dtype == np.float32 else np.uint64))


def _check(run, s, m):
    s, m = (np.ascontiguousarray(a, np.float64) for a in np.broadcast_arrays(s, m))
    with np.errstate(all="ignore"):
        want = (s / m).astype(np.float32)
        f = m.astype(np.float32)
    q, w = run(s, m, f)
    bad = ~((q.view(np.uint32) == want.view(np.uint32)) | (np.isnan(q) & np.isnan(want)))
    assert not bad.any(), (s[bad][:3], m[bad][:3], q[bad][:3], want[bad][:3])
    assert _same(w, f.astype(np.float64))


def _masses(rng, n):
    return rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(-50, 50, n)


@pytest.mark.parametrize("steps", [0, 1, 2, 3, 8, 1000, 1 << 14, 1 << 17])
def test_around_the_middle_of_two_floats(run, steps):
    """s within a few units in the last place of (middle of two floats) x m, and within
    the 2^-38 that the guard leaves to the division."""
    rng = np.random.default_rng(steps)
    n = 200000
    m = _masses(rng, n)
    f = (rng.uniform(-2.0, 2.0, n) * 2.0 ** rng.integers(-40, 10, n)).astype(np.float32)
    mid = 0.5 * (f.astype(np.float64) + np.nextafter(f, np.float32(np.inf)).astype(np.float64))
    s = mid * m
    bits = s.view(np.int64) + rng.integers(-steps, steps + 1, n)
    _check(run, bits.view(np.float64), m)


def test_around_powers_of_two_and_floats(run):
    rng = np.random.default_rng(1)
    n = 200000
    m = _masses(rng, n)
    for base in (2.0 ** rng.integers(-59, 60, n), rng.uniform(1, 2, n).astype(np.float32).astype(np.float64)):
        for step in (0, 1, -1, 3, 1 << 28, -(1 << 28), (1 << 29) - 1, 1 << 14):
            s = ((base * m).view(np.int64) + step).view(np.float64)
            _check(run, np.where(rng.random(n) < 0.5, s, -s), m)


def test_the_whole_range(run):
    rng = np.random.default_rng(2)
    n = 400000
    s = rng.uniform(-2, 2, n) * 2.0 ** rng.integers(-200, 200, n)
    m = rng.uniform(-2, 2, n) * 2.0 ** rng.integers(-200, 200, n)
    _check(run, s, m)
    _check(run, s * 2.0 ** -900, m)  # down to subnormal sums
    edge = 2.0 ** np.array([-1074., -1022., -150., -149., -126., -61., -60., 60., 61., 127., 128., 1000.])
    v = np.concatenate([edge, -edge, edge * (1 + 2.0 ** -52), edge * (1 - 2.0 ** -53), [0.0, -0.0, np.inf, -np.inf, np.nan]])
    a, b = np.meshgrid(v, v)
    _check(run, a.ravel(), b.ravel())


def test_random_sums_of_a_cell(run):
    """Sums as cells have them: up to eight bodies' m x over m."""
    rng = np.random.default_rng(3)
    n = 300000
    m = rng.uniform(0.1, 2.0, (8, n)).astype(np.float32).astype(np.float64)
    x = rng.normal(size=(8, n)).astype(np.float32).astype(np.float64)
    _check(run, (m * x).sum(0), m.sum(0))
