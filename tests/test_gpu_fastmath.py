"""The arithmetic of gpr_fastmath.cuh against exact values and CUDA's own
operators, by a kernel compiled from the header.

Bars, in units in the last place of the exact value (u = 2^-53, so half a unit
is at most u relative).  rcp64: one rounding (1/2) and the truncation of the
geometric series at e^3, e = 2^-19.9, at most 2 e^3 / 2^-52 = 0.02.  sqrt64:
one rounding and the root's error 2^-39 times the reciprocal root's 2^-20:
0.02.  rsqrt64: the rounding of x y (half a unit through the square root's
factor 1/2, doubled by the scale of the unit) and the last one: 1, and 0.05 for
5/16 e^3.  pow53: the roundings of x |x|, its product with y and the last one
(u each), a third of the one in e, and the truncation: 3.4 u, so 3.4 units.
Zeros, infinities, NaNs, subnormals and what else lies outside a form's range
take CUDA's operator, bit for bit."""
import ctypes
import os
import subprocess
from decimal import Decimal, getcontext
from fractions import Fraction

import numpy as np
import pytest
import torch

from conftest import ROOT

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

SRC = r"""
#include "gpr_kernels.cuh"
using namespace gpr;
__global__ void k(int f, const double *x, double *o, double *ref, long n, int sh) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  const double v = x[i];
  double a = 0.0, r = 0.0;
  if (f == 0) { a = rcp64(v); r = 1.0 / v; }
  if (f == 1) { a = sqrt64(v); r = sqrt(v); }
  if (f == 2) { a = rsqrt64(v); r = rsqrt(v); }
  if (f == 3) { a = pow53(v); const double c = cbrt(v); r = v * c * c; }
  if (f == 4) { a = f32_scaled(v, sh); r = f64_scaled((float)a, sh); }
  if (f == 5) { a = f32_abs_hi(v); r = v; }
  o[i] = a;
  ref[i] = r;
}
extern "C" int run(int f, const double *x, double *o, double *ref, long n, int sh) {
  k<<<(unsigned)((n + 127) / 128), 128>>>(f, x, o, ref, n, sh);
  return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def lib(cuda_ok, tmp_path_factory):
    from phd_gb300 import _lib
    d = tmp_path_factory.mktemp("fastmath")
    src, so = os.path.join(d, "f.cu"), os.path.join(d, "f.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run([os.environ.get("NVCC", "nvcc")] + _lib.ARCH +
                   ["-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-I", _lib.CSRC,
                    "-I", os.path.join(ROOT, "include"), src, "-o", so], check=True)
    return ctypes.CDLL(so)


def _run(lib, f, x, sh=0):
    t = torch.tensor(np.ascontiguousarray(x, dtype=np.float64), device=DEV)
    o, r = torch.empty_like(t), torch.empty_like(t)
    p = [ctypes.c_void_p(a.data_ptr()) for a in (t, o, r)]
    torch.cuda.synchronize()
    assert lib.run(f, p[0], p[1], p[2], ctypes.c_long(t.numel()), sh) == 0
    return o.cpu().numpy(), r.cpu().numpy()


def _numbers(lo, hi, n, seed, negative=False):
    """n numbers of random mantissa and exponents uniform in [lo, hi]."""
    rng = np.random.default_rng(seed)
    x = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(lo, hi + 1, n))
    return x * rng.choice([-1.0, 1.0], n) if negative else x


def _ulp(x):
    return Fraction(float(np.spacing(abs(x))))


EDGES = [0.0, -0.0, 5e-324, -5e-324, 2.2e-308, 2.2250738585072014e-308, -2.2250738585072014e-308,
         1.7976931348623157e308, -1.7976931348623157e308, np.inf, -np.inf, np.nan]


def _same(a, b):
    return np.array_equal(a.view(np.int64)[~np.isnan(a)], b.view(np.int64)[~np.isnan(a)]) and \
        np.array_equal(np.isnan(a), np.isnan(b))


def test_reciprocal(lib):
    x = _numbers(-1022, 1021, 1 << 20, 1, True)
    got, ref = _run(lib, 0, x)
    assert np.max(np.abs(got.view(np.int64) - ref.view(np.int64))) <= 1
    for b, r in zip(x[:4096], got[:4096]):
        assert abs(Fraction(r) - 1 / Fraction(b)) <= Fraction(52, 100) * _ulp(1 / b)
    # the operator's: the ends of the range (a reciprocal below 2^-1022 among them)
    x = np.array(EDGES + list(_numbers(-1074, -1024, 64, 2, True)) +
                 list(np.ldexp(1.0 + 0.01 * np.arange(1, 64), 1022)))
    got, ref = _run(lib, 0, x)
    assert _same(got, ref)
    # powers of two are exact
    x = np.ldexp(1.0, np.arange(-1021, 1022))
    assert np.array_equal(_run(lib, 0, x)[0], 1.0 / x)


def test_square_root(lib):
    x = _numbers(-899, 1023, 1 << 20, 3)
    got, ref = _run(lib, 1, x)
    assert np.max(np.abs(got.view(np.int64) - ref.view(np.int64))) <= 1
    for v, r in zip(x[:4096], got[:4096]):
        # |r - sqrt v| <= h  <=>  (r - h)^2 <= v <= (r + h)^2
        h = Fraction(52, 100) * _ulp(float(np.sqrt(v)))
        assert (Fraction(r) - h) ** 2 <= Fraction(v) <= (Fraction(r) + h) ** 2
    x = np.array(EDGES + [-1.0, -1e-300] + list(_numbers(-1074, -901, 256, 4)))
    x = x[x != np.finfo(np.float64).max]  # within the form's range
    got, ref = _run(lib, 1, x)
    assert _same(got, ref)
    # squares are exact
    k = np.arange(1.0, 4097.0)
    assert np.array_equal(_run(lib, 1, k * k)[0], k)


def test_reciprocal_root(lib):
    x = _numbers(-900, 900, 1 << 20, 5)
    got, ref = _run(lib, 2, x)
    assert np.max(np.abs(got.view(np.int64) - ref.view(np.int64))) <= 3
    for v, r in zip(x[:4096], got[:4096]):
        h = Fraction(105, 100) * _ulp(float(1 / np.sqrt(v)))
        assert (Fraction(r) - h) ** 2 * Fraction(v) <= 1 <= (Fraction(r) + h) ** 2 * Fraction(v)


def test_power_five_thirds(lib):
    getcontext().prec = 50
    x = _numbers(-300, 299, 2048, 6, True)
    x = np.concatenate([x, _numbers(-3, 3, 2048, 7)])
    got, ref = _run(lib, 3, x)
    for v, r in zip(x, got):
        e = Decimal(abs(float(v))) ** (Decimal(5) / 3)
        assert np.sign(r) == np.sign(v)
        assert abs(Decimal(abs(float(r))) - e) <= Decimal("3.4") * Decimal(float(np.spacing(float(e))))
    x = np.array(EDGES + list(_numbers(-1074, -301, 256, 8, True)) +
                 list(_numbers(301, 612, 256, 9, True)))
    got, ref = _run(lib, 3, x)
    assert _same(got, ref)


@pytest.mark.parametrize("sh", [-240, -1, 0, 3, 240])
def test_bit_field_conversions(lib, sh):
    x = np.ldexp(_numbers(-126, 126, 1 << 16, 10, True), sh)
    got, back = _run(lib, 4, x, sh)
    cut = (x.view(np.int64) & ~((1 << 29) - 1)).view(np.float64)  # to 24 bits, towards zero
    assert np.array_equal(back, cut)
    assert np.array_equal(np.ldexp(got, sh), cut)
    low = np.ldexp(_numbers(-200, -127, 256, 11, True), sh)
    assert np.all(_run(lib, 4, low, sh)[0] == 0)
    assert np.all(_run(lib, 4, np.array([0.0, -0.0, 5e-324]), sh)[0] == 0)
    high = np.ldexp(_numbers(128, 200, 256, 12, True), sh)
    high = np.concatenate([high, [np.inf, -np.inf, np.nan]])
    assert np.all(~(np.abs(_run(lib, 4, high, sh)[0]) < 2.0 ** 127))


def test_high_word_magnitude(lib):
    x = _numbers(-126, 126, 1 << 16, 13, True)
    got = _run(lib, 5, x)[0]
    assert np.all(got <= np.abs(x)) and np.all(got > np.abs(x) * (1 - 2.0 ** -20))
    assert np.all(_run(lib, 5, _numbers(-300, -127, 256, 14))[0] == 0)
    assert np.all(_run(lib, 5, np.array([0.0, -0.0, 5e-324]))[0] == 0)
    big = np.concatenate([_numbers(127, 300, 256, 15, True), [np.inf, -np.inf, np.nan]])
    assert np.all(_run(lib, 5, big)[0] == 2.0 ** 127)
