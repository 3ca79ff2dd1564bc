"""The FP64 kernels' stand-ins for plain operations, bit for bit against those operations: quotients by a shared divisor
(and by c and 2c) against IEEE division, uniform deviates put together from integers, and the cosine that is taken
without its sine."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from spectrum_gb300 import build, units

pytestmark = pytest.mark.gpu

QUOT, OVER_C, OVER_2C, UNIFORM = range(4)


@pytest.fixture(scope="module")
def device(tmp_path_factory):
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "device_arithmetic.cu")
    out = str(tmp_path_factory.mktemp("arithmetic") / "libarithmetic.so")
    subprocess.run([build._nvcc(), *build.ARCH, *build.CFLAGS, "-fmad=false", "-I", build.CSRC, "-shared", "-o", out, src], check=True)
    return ctypes.CDLL(out)


def _apply(device, op, x=None, y=None, u=None):
    n = len(x if u is None else u)
    out = np.empty(n)
    p = lambda a, t: None if a is None else np.ascontiguousarray(a).ctypes.data_as(ctypes.POINTER(t))  # noqa: E731
    assert device.arithmetic(op, ctypes.c_int64(n), p(x, ctypes.c_double), p(y, ctypes.c_double), p(u, ctypes.c_uint32),
                             p(out, ctypes.c_double)) == 0
    return out


def _same(got, want):
    assert np.array_equal(np.isnan(got), np.isnan(want))
    k = ~np.isnan(want)
    assert np.array_equal(got[k].view(np.int64), want[k].view(np.int64))


def _doubles(exponents, significands):
    """Doubles of all biased exponents x 52-bit significands, in both signs."""
    e, m = np.meshgrid(np.array(exponents, np.uint64), np.array(significands, np.uint64))
    v = ((e << np.uint64(52)) | m).ravel().view(np.float64)
    return np.concatenate([v, -v])


# exponents on both sides of the windows of divisor (623 .. 1422) and dividend (523 .. 1522), zero and subnormal
# numbers (0), the largest (2046), infinities and NaN (2047); significands at both ends and in the middle
EDGES = _doubles([0, 1, 522, 523, 524, 622, 623, 624, 1022, 1023, 1422, 1423, 1424, 1521, 1522, 1523, 2045, 2046, 2047],
                 [0, 1, 2, 2 ** 51, 2 ** 52 - 2, 2 ** 52 - 1])


def _beside_midpoints(n, seed):
    """Dividends and divisors whose quotient is as near as can be to the middle m / 2 of two doubles: m y = x 2^k + d with a
    small odd d, m an odd number of 54 bits. Every second divisor is just below a power of two."""
    r = np.random.default_rng(seed)
    x, y = [], []
    for a, near, d in zip(r.integers(2 ** 52, 2 ** 53, n).tolist(), r.integers(1, 10 ** 7, n).tolist(), r.integers(-8, 8, n).tolist()):
        for div in (a | 1, 2 ** 53 - (near | 1)):
            for k in (53, 54):
                m = (2 * d + 1) * pow(div, -1, 1 << k) % (1 << k)
                m += (m < 2 ** 53) << 53  # (k = 53: the one of 54 bits)
                q, rest = divmod(m * div - (2 * d + 1), 1 << k)
                if rest == 0 and 2 ** 52 <= q < 2 ** 53:
                    x.append(float(q))
                    y.append(float(div))
    return np.array(x), np.array(y)


def test_quotients_equal_division(device):
    r = np.random.default_rng(5)
    ex, ey = (a.ravel() for a in np.meshgrid(EDGES, EDGES))
    bits = r.integers(0, 2 ** 64, (2, 1 << 21), dtype=np.uint64).view(np.float64)  # every exponent, infinities and NaN
    ones = r.uniform(1.0, 2.0, (2, 1 << 21))
    mx, my = _beside_midpoints(50_000, 6)
    x, y = np.concatenate([ex, bits[0], ones[0], mx, EDGES]), np.concatenate([ey, bits[1], ones[1], my, np.ones_like(EDGES)])
    with np.errstate(all="ignore"):
        _same(_apply(device, QUOT, x, y), x / y)


@pytest.mark.parametrize("op,factor", [(OVER_C, 1.0), (OVER_2C, 2.0)])
def test_quotients_by_the_speed_of_light(device, op, factor):
    r = np.random.default_rng(7)
    c = factor * units.c_code
    mx, _ = _beside_midpoints(1000, 8)
    x = np.concatenate([EDGES, mx, r.integers(0, 2 ** 64, 1 << 20, dtype=np.uint64).view(np.float64), r.uniform(1.0, 2.0, 1 << 20)])
    with np.errstate(all="ignore"):
        _same(_apply(device, op, x), x / c)


def test_uniform_deviates(device):
    k = 2 ** np.arange(32, dtype=np.uint64)
    x = np.concatenate([[0, 2 ** 32 - 1], k, k - 1, k + 1, np.random.default_rng(9).integers(0, 2 ** 32, 1 << 20)]).astype(np.uint32)
    _same(_apply(device, UNIFORM, u=x), (x.astype(np.float64) + 0.5) * 2.0 ** -32)


def test_cosine_without_its_sine(device):
    n = ctypes.c_ulonglong(1)
    assert device.cosines_that_differ(ctypes.byref(n)) == 0 and n.value == 0
