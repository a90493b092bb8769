"""Quotients by series (nyles_div.cuh) beside CUDA's own division, over the divisors that the right-hand side by lines
forms: products of three smoothness indicators, from 6.4e-46 up to the end of the range.

Bars: the seed within 2^-20 + 2^-22 of 1/x, for which the series leaves e^3 < 2^-59; two roundings of 2^-53 and that
remainder are at most 2 units in the last place from a correctly rounded quotient (2^-52 is 2 units at the top of
a binade, and a distance of whole units).
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SRC = r"""
#include "nyles_div.cuh"
__global__ void k(const double* a, const double* x, double* q, double* ref, double* seed, long long n) {
    const long long i = blockIdx.x * 256ll + threadIdx.x;
    if (i >= n) return;
    q[i] = nyles::div_series(a[i], x[i]);
    ref[i] = a[i] / x[i];
    seed[i] = fma(-x[i], nyles::div_seed(x[i]), 1.0);
}
extern "C" int run(const double* a, const double* x, double* q, double* ref, double* seed, long long n) {
    k<<<(unsigned)((n + 255) / 256), 256>>>(a, x, q, ref, seed, n);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def div(tmp_path_factory):
    from nyles_gb300 import build
    d = tmp_path_factory.mktemp("div")
    (d / "div.cu").write_text(SRC)
    r = subprocess.run([build.nvcc(), "-shared", str(d / "div.cu"), "-o", str(d / "libdiv.so"), "-I" + build.CSRC] + build.ARCH +
                       build.FLAGS, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    lib = ctypes.CDLL(os.path.join(str(d), "libdiv.so"))

    def run(a, x):
        t = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (a, x)]
        t += [torch.empty_like(t[0]) for _ in range(3)]
        assert lib.run(*[ctypes.c_void_p(v.data_ptr()) for v in t], ctypes.c_longlong(a.size)) == 0
        return [v.cpu().numpy() for v in t[2:]]
    return run


def _check(div, a, x):
    q, ref, seed = div(a, x)
    assert np.isfinite(ref).all()
    assert np.abs(seed).max() <= 2.0 ** -20 + 2.0 ** -22, np.abs(seed).max() * 2.0 ** 20
    units = np.abs(q.view(np.int64) - ref.view(np.int64))
    assert units.max() <= 2, (units.max(), a[units.argmax()], x[units.argmax()])


def test_every_leading_mantissa_bit_pattern(div):
    """2^21 mantissas evenly over a binade with random low bits"""
    rng = np.random.Generator(np.random.PCG64(1))
    x = 1.0 + (np.arange(1 << 21) + rng.uniform(0, 1, 1 << 21)) / (1 << 21)
    _check(div, np.ones_like(x), x)
    _check(div, rng.uniform(-2, 2, x.size), x)


@pytest.mark.parametrize("lo,hi", [(-151.0, 0.0), (0.0, 400.0), (400.0, 1021.9)])
def test_range_of_the_divisors(div, lo, hi):
    """divisors from 2^-151 (6.4e-46 is 2^-150.2) on, quotients of the size of the field's differences"""
    rng = np.random.Generator(np.random.PCG64(2))
    x = np.exp2(rng.uniform(lo, hi, 1 << 20)) * rng.uniform(1.0, 1.05, 1 << 20)
    _check(div, x * 0.9 * rng.uniform(-1, 1, x.size), x)
    ends = np.array([6.4e-46, np.nextafter(1.0, 0), 1.0, np.nextafter(1.0, 2), 2.0 - 2.0 ** -52, 2.0 ** 1021])
    _check(div, np.ones_like(ends), ends)
