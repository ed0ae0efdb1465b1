"""IEEE double operations on the integer pipe (csrc/intfp64.h), compiled for the
host and checked against the host's own FP64 arithmetic: products, quotients
and roots bit for bit, logarithms and reciprocal roots to a fraction of an ulp.
The FP32 estimates that the device takes from its special-function unit are off
by up to 2^-22; the host's are moved by up to three FP32 ulps either way."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include "intfp64.h"
// b / sqrt(a) by ip_rroot64's significand (2^63 to 2^64)
struct ip_factor {
    ip_u64 r;
    int e;
};

static inline ip_factor ip_rsqrt_fit(double x)
{
    const ip_u64 u = ip_bits(x);
    const int e = ip_exponent(u);
    const uint32_t s = (uint32_t)e & 1u;
    const ip_u64 M = ((u & IP_FRACTION) | IP_IMPLICIT) << (11 - s);
    const uint32_t Y =
        ip_estimate(((126u - s) << 23) | ((uint32_t)(u >> 29) & 0x7fffffu), true);
    ip_factor f;
    f.r = ip_rroot64(M, Y);
    f.e = (1023 * 3 - 1 - e + (int)(1u - s)) >> 1;
    return f;
}

/* a * f, within 0.51 ulp, of an operand that fits */
static inline double ip_apply_fit(double a, const ip_factor& f)
{
    const ip_u64 u = ip_bits(a);
    ip_u64 q = ip_mulhi(ip_left(u), f.r);
    int e = ip_exponent(u) + f.e - 1022;
    if (!(q >> 63)) {
        q <<= 1;
        e -= 1;
    }
    return ip_pack(u, (q >> 11) + ((q >> 10) & 1), e);
}
extern "C" {
void t_mul(const double* a, const double* b, long n, double* o) { for (long i = 0; i < n; ++i) o[i] = ip_mul(a[i], b[i]); }
void t_div(const double* a, const double* b, long n, double* o) { for (long i = 0; i < n; ++i) o[i] = ip_div(a[i], ip_reciprocal(b[i])); }
void t_sub(const double* a, const double* b, long n, double* o) { for (long i = 0; i < n; ++i) o[i] = ip_sub(a[i], b[i]); }
void t_sqrt(const double* a, const double*, long n, double* o) { for (long i = 0; i < n; ++i) o[i] = ip_sqrt(a[i]); }
void t_log(const double* a, const double*, long n, double* o) { for (long i = 0; i < n; ++i) o[i] = ip_log(a[i]); }
void t_sin(const double* a, const double*, long n, double* o) { for (long i = 0; i < n; ++i) { double c; ip_sincos(a[i], o + i, &c); if (ip_bits(o[i]) != ip_bits(ip_sin(a[i]))) o[i] = 99.0; } }
void t_cos(const double* a, const double*, long n, double* o) { for (long i = 0; i < n; ++i) { double s; ip_sincos(a[i], &s, o + i); } }
void t_rsqrt(const double* a, const double* b, long n, double* o) { for (long i = 0; i < n; ++i) o[i] = ip_apply_fit(b[i], ip_rsqrt_fit(a[i])); }
}
"""


@pytest.fixture(scope="module", params=[0, -3, 3])
def lib(request, tmp_path_factory):
    d = tmp_path_factory.mktemp("intfp64")
    src, out = d / "t.cpp", d / "t.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off",
                    "-DNBCS_INTFP64_ESTIMATE_ULPS=(%d)" % request.param,
                    "-I", os.path.join(ROOT, "numbacs_gb300", "csrc"), str(src), "-o", str(out)],
                   check=True)
    return ctypes.CDLL(str(out))


def _call(lib, name, a, b):
    o = np.empty_like(a)
    p = ctypes.POINTER(ctypes.c_double)
    getattr(lib, name)(a.ctypes.data_as(p), b.ctypes.data_as(p), ctypes.c_long(len(a)),
                       o.ctypes.data_as(p))
    return o


def _bits(a):
    return a.view(np.uint64)


def _numbers(rng, n, lo, hi):
    """Doubles of exponents [lo, hi): a part with short significands, all ones
    or a single one, where quotients and roots come out exact or next to it."""
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    k = rng.integers(0, 8, n)
    m[k == 0] = 0
    m[k == 1] = (1 << 52) - 1
    cut = rng.integers(1, 52, n, dtype=np.uint64)
    low = (np.uint64(1) << cut) - np.uint64(1)
    m = np.where(k == 2, m & ~low, m)
    m = np.where(k == 3, m | low, m)
    m = np.where(k == 4, m & np.uint64(15), m)
    e = (rng.integers(lo, hi, n) + 1023).astype(np.uint64)
    s = rng.integers(0, 2, n, dtype=np.uint64)
    return ((s << np.uint64(63)) | (e << np.uint64(52)) | m).view(np.float64)


EDGES = np.array([0.0, -0.0, 5e-324, 2.2250738585072014e-308, 2.0 ** -256, 2.0 ** -255, 2.0 ** 255,
                  np.nextafter(2.0 ** 256, 0), 2.0 ** 256, 1.7976931348623157e308, np.inf, -np.inf,
                  np.nan, 1.0, np.nextafter(1.0, 0), np.nextafter(1.0, 2), 2.0, 3.0, -1.0 / 3.0])


def _pairs(span):
    rng = np.random.default_rng(5)
    a, b = _numbers(rng, 200000, -span, span), _numbers(rng, 200000, -span, span)
    g = np.meshgrid(EDGES, EDGES, indexing="ij")
    return (np.concatenate([a, a * b, g[0].ravel()]), np.concatenate([b, b, g[1].ravel()]))


@pytest.mark.parametrize("span", [2, 120, 255])
def test_products_quotients_roots_bit_for_bit(lib, span):
    a, b = _pairs(span)
    with np.errstate(all="ignore"):
        for name, want in (("t_mul", a * b), ("t_div", a / b)):
            got = _call(lib, name, a, b)
            nan = np.isnan(want)
            assert np.array_equal(np.isnan(got), nan), name
            assert np.array_equal(_bits(got)[~nan], _bits(want)[~nan]), name
        # differences of neighbours: the same exponent, the next one, the next double
        near = ((a.view(np.uint64) & ~np.uint64((1 << 52) - 1)) |
                (b.view(np.uint64) & np.uint64((1 << 52) - 1))).view(np.float64)
        for c in (b, near, near * 2.0, near * 0.5, a, np.nextafter(a, b), -near):
            want, got = a - c, _call(lib, "t_sub", a, c)
            nan = np.isnan(want)
            assert np.array_equal(np.isnan(got), nan)
            assert np.array_equal(_bits(got)[~nan], _bits(want)[~nan])
        for x in (a, a * a, np.nextafter(a * a, np.inf)):
            want, got = np.sqrt(x), _call(lib, "t_sqrt", x, x)
            nan = np.isnan(want)
            assert np.array_equal(np.isnan(got), nan)
            assert np.array_equal(_bits(got)[~nan], _bits(want)[~nan])


def _ulps(got, want):
    """|got - want| in ulps of want (a long double)."""
    ulp = np.ldexp(1.0, np.frexp(want.astype(np.float64))[1] - 53)
    return np.abs(got.astype(np.longdouble) - want) / ulp


@pytest.mark.skipif(np.finfo(np.longdouble).nmant < 63, reason="needs an 80-bit long double")
def test_logarithm_and_reciprocal_root(lib):
    rng = np.random.default_rng(6)
    x = np.concatenate([1.0 + rng.random(100000) * s for s in (1e-12, 0.01, 1.0)] +
                       [np.exp(rng.random(100000) * 160.0), 1.0 + np.arange(1, 513) / 256.0,
                        [np.nextafter(1.0, 2), np.nextafter(2.0, 1), 2.0, np.nextafter(2.0 ** 256, 0),
                         2.0 ** 256, 1e300]])
    # half an ulp of rounding, 2^-60 relative of fixed point and series
    assert _ulps(_call(lib, "t_log", x, x), np.log(x.astype(np.longdouble))).max() < 0.55
    a = np.abs(_numbers(rng, 200000, -200, 200))
    b = _numbers(rng, 200000, -200, 200)
    want = b.astype(np.longdouble) / np.sqrt(a.astype(np.longdouble))
    assert _ulps(_call(lib, "t_rsqrt", a, b), want).max() < 0.55


@pytest.mark.skipif(np.finfo(np.longdouble).nmant < 63, reason="needs an 80-bit long double")
def test_sine_and_cosine(lib):
    rng = np.random.default_rng(7)
    x = np.concatenate([rng.uniform(-64, 64, 200000), rng.uniform(-2, 2, 100000),
                        np.exp(rng.uniform(-60, 4, 100000)),
                        np.arange(-80, 81) * (np.pi / 4), np.arange(-40, 41) * (np.pi / 2) * (1 + 1e-12),
                        [0.0, -0.0, 2.0 ** -27, -(2.0 ** -27), np.nextafter(64.0, 0), 64.0, -100.0,
                         1e300]])
    for name, fn in (("t_sin", np.sin), ("t_cos", np.cos)):
        got, want = _call(lib, name, x, x), fn(x.astype(np.longdouble))
        # a rounding (0.5 ulp and the series' 2^-60) plus the reduction's 2^-58
        # absolute; below 2^-27 the argument itself (half an ulp off), and the
        # library beyond 64 (within an ulp)
        ulp = np.ldexp(1.0, np.frexp(want.astype(np.float64))[1] - 53)
        err = np.abs(got.astype(np.longdouble) - want)
        slack = np.where(np.abs(x) < 0.75, 0.0, 2.0 ** -58)
        assert np.all(err <= np.where(np.abs(x) < 64, 0.52, 1.0) * ulp + slack), name
    assert np.all(np.isnan(_call(lib, "t_sin", np.array([np.inf, np.nan]), np.zeros(2))) |
                  (_call(lib, "t_sin", np.array([np.inf, np.nan]), np.zeros(2)) == 99.0))
    z = _call(lib, "t_sin", np.array([0.0, -0.0]), np.zeros(2))
    assert np.array_equal(np.signbit(z), [False, True]) and not z.any()


@pytest.mark.parametrize("apart", range(-11, 12))
def test_differences_of_every_gap(lib, apart):
    """exponents up to nine apart and beyond, both signs, low bits that make
    ties: the same bits as the hardware's"""
    rng = np.random.default_rng(100 + apart)
    a = np.ldexp(rng.uniform(1.0, 2.0, 20000), rng.integers(-40, 40, 20000))
    b = np.ldexp(rng.uniform(1.0, 2.0, 20000), np.frexp(a)[1] - 1 - apart)
    keep = np.uint64(0xffffffffffffffff) << rng.integers(0, 53, 20000).astype(np.uint64)
    for x, y in ((a, b), (a, (b.view(np.uint64) & keep).view(np.float64)),
                 ((a.view(np.uint64) & keep).view(np.float64), b),
                 (a, (b.view(np.uint64) | ~keep & np.uint64((1 << 52) - 1)).view(np.float64))):
        for s in (1.0, -1.0):
            for t in (1.0, -1.0):
                assert np.array_equal(_bits(_call(lib, "t_sub", s * x, t * y)), _bits(s * x - t * y))
