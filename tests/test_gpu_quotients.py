"""Quotients formed without the division must be the division's, bit for bit.

div3 (three numerators over one density, one division for all), min_image (a
lattice offset wrapped without one) and recip_ge1 (the sigmoid's reciprocal) say
so beside their code. The FP64 ones are compared with IEEE division on the host:
ordinary values, values of every exponent, zeros of both signs, the smallest and
largest numbers, infinities and NaN, and both sides of the exponents where div3
leaves the quick way. They are built with and without FMA contraction, as the
library's forms are. The reciprocal is compared over every float of its range
and the special values beyond it.
"""
import ctypes
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

NVCC = "/usr/local/cuda/bin/nvcc"


def native(tmp, source, *flags):
    out = tmp / "probe.so"
    subprocess.run([NVCC, "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC",
                    "--expt-relaxed-constexpr", "-shared", *flags, str(ROOT / "tests" / "native" / source), "-o", str(out)],
                   check=True)
    return ctypes.CDLL(str(out))


@pytest.fixture(scope="module", params=["--fmad=false", "--fmad=true"])
def quotients(request, tmp_path_factory):
    return native(tmp_path_factory.mktemp("quot"), "quotients.cu", request.param)


def ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def same(x, y):
    return np.array_equal(np.where(np.isnan(x), 0, x).view(np.uint64), np.where(np.isnan(y), 0, y).view(np.uint64)) and \
        np.array_equal(np.isnan(x), np.isnan(y))


def of_exponents(rng, n, lo, hi):
    """Doubles with random mantissas and signs and binary exponents in [lo, hi]."""
    return np.ldexp(rng.uniform(1.0, 2.0, n) * rng.choice([-1.0, 1.0], n), rng.integers(lo, hi + 1, n))


EDGES = np.array([0.0, -0.0, 1.0, -1.0, 1.0 / 3.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.2250738585072014e-308,
                  1.7976931348623157e308] +
                 [s * np.ldexp(m, e) for e in (-514, -513, -512, -511, -501, -500, -499, 498, 499, 500, 501, 510, 511, 512)
                  for m in (1.0, 1.3333333333333333, 1.9999999999999998) for s in (1.0, -1.0)])


def div3(lib, a, b):
    a, b = np.ascontiguousarray(a, np.float64), np.ascontiguousarray(b, np.float64)
    q = np.empty_like(a)
    assert lib.quot_div3(ptr(a), ptr(b), ptr(q), ctypes.c_size_t(b.size)) == 0
    return q


def test_div3(quotients):
    rng = np.random.default_rng(1)
    n = 1 << 21
    sets = [(rng.normal(size=(n, 3)) * 0.1, rng.uniform(0.5, 1.5, n)),                # momenta over densities
            (of_exponents(rng, 3 * n, -60, 60).reshape(n, 3), of_exponents(rng, n, -60, 60)),
            (of_exponents(rng, 3 * n, -1074, 1023).reshape(n, 3), of_exponents(rng, n, -1074, 1023)),
            (of_exponents(rng, 3 * n, -514, -498).reshape(n, 3), of_exponents(rng, n, 498, 513)),
            (of_exponents(rng, 3 * n, 498, 513).reshape(n, 3), of_exponents(rng, n, -514, -498))]
    e = EDGES.size
    a, b = np.repeat(EDGES, e), np.tile(EDGES, e)
    # an edge beside ordinary numerators and two other edges
    sets += [(np.stack([a, np.full(e * e, 0.3), np.full(e * e, -0.0)], 1), b),
             (np.stack([np.full(e * e, 0.25), a, np.roll(a, 7)], 1), b),
             (np.stack([np.zeros(e), -np.zeros(e), EDGES], 1), np.full(e, 0.97))]
    with np.errstate(all="ignore"):
        for a, b in sets:
            assert same(div3(quotients, a, b), a / b[:, None])


def test_min_image(quotients):
    rng = np.random.default_rng(2)
    n = 1 << 21
    m = rng.integers(1, 1200, n).astype(np.int32)
    spread = [0.5, 0.4995, 1.0, 3.0, 1e4, 1e9]
    r = np.concatenate([rng.uniform(-s, s, n // 8) for s in spread] + [rng.integers(-8, 9, n // 8) * 0.5,
                       (rng.integers(-8, 9, n - 7 * (n // 8)) + 0.5) * (1.0 + rng.integers(-2, 3, n - 7 * (n // 8)) * 2.0 ** -52)])
    r = np.ascontiguousarray(r * m)
    r[:8] = [0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1e300, -1e300]
    t = np.empty(n)
    assert quotients.quot_min_image(ptr(r), ptr(m), ptr(t), ctypes.c_size_t(n)) == 0
    with np.errstate(all="ignore"):
        x = r / m
        k = np.trunc(x)
        k = np.where(np.abs(x - k) >= 0.5, k + np.sign(x), k)   # round(), halves away from zero
        small = np.abs(k) < 2.0 ** 40                           # m k exact
        want = r - m * k
    assert same(t[small | ~np.isfinite(r)], want[small | ~np.isfinite(r)])


def test_recip(tmp_path):
    lib = native(tmp_path, "recip.cu")
    wrong = ctypes.c_ulonglong(0)

    def count(first, n):
        assert lib.recip_wrong(ctypes.c_uint(first), ctypes.c_ulonglong(n), ctypes.byref(wrong)) == 0
        return wrong.value

    one, two100 = 0x3F800000, (127 + 100) << 23
    assert count(one, two100 - one) == 0                  # every float in [1, 2^100)
    assert count(two100, 0x7F800000 - two100 + 16) == 0   # up to infinity, and NaN
