"""Sine and cosine on the integer pipe (csrc/intfp64.h) next to their zeros, where
the reduced angle is many orders below the argument: against the difference to
the zero, taken with 80 digits of pi."""
import ctypes
import math
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PI = Fraction(31415926535897932384626433832795028841971693993751058209749445923078164062862089,
              10 ** 79)

SRC = r"""
#include "intfp64.h"
extern "C" void t_sincos(const double* a, long n, double* s, double* c, double* s1)
{
    for (long i = 0; i < n; ++i) {
        ip_sincos(a[i], s + i, c + i);
        s1[i] = ip_sin(a[i]);
    }
}
"""


@pytest.fixture(scope="module")
def sincos(tmp_path_factory):
    d = tmp_path_factory.mktemp("intfp64z")
    src, out = d / "t.cpp", d / "t.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "numbacs_gb300", "csrc"), str(src), "-o", str(out)],
                   check=True)
    lib = ctypes.CDLL(str(out))

    def call(x):
        o = [np.empty_like(x) for _ in range(3)]
        p = ctypes.POINTER(ctypes.c_double)
        lib.t_sincos(x.ctypes.data_as(p), ctypes.c_long(len(x)), *[v.ctypes.data_as(p) for v in o])
        return o

    return call


def _near_zero(x, k):
    """sin(x) for k even, cos(x) for k odd, x next to k pi / 2: the Taylor series
    of the difference, exact to 1e-40 of it"""
    d = Fraction(x) - k * PI / 2
    s = d * (1 - d * d / 6 * (1 - d * d / 20 * (1 - d * d / 42 * (1 - d * d / 72))))
    return s * (1, -1, -1, 1)[k % 4]


@pytest.mark.parametrize("off", [0.0, 1e-15, 1e-13, 1e-10, 1e-7, 1e-5, 1e-3])
def test_next_to_every_zero(sincos, off):
    ks, xs = [], []
    for k in range(1, 41):
        x = k * math.pi / 2 * (1.0 + off)
        for step in range(-3, 4):
            y = x
            for _ in range(abs(step)):
                y = math.nextafter(y, math.inf * step)
            if y < 64.0:
                ks += [k, -k]
                xs += [y, -y]
    s, c, s1 = sincos(np.array(xs))
    assert np.array_equal(s, s1)
    for k, x, sv, cv in zip(ks, xs, s, c):
        got, want = (sv, cv)[k % 2], _near_zero(x, k)
        assert abs(Fraction(float(got)) - want) <= Fraction(0.52) * Fraction(math.ulp(float(want))), (k, x)
