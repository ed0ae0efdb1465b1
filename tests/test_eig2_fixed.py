"""Eigenvalue and eigenvector of the fused FTLE kernel (csrc/eig2_fixed.h), compiled
for the host: gradients of any ratio against 80-bit arithmetic, and never further
off than the FP64 operations of the general form."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
U = 2.0 ** -53

pytestmark = pytest.mark.skipif(np.finfo(np.longdouble).nmant < 63,
                                reason="needs an 80-bit long double")

SRC = r"""
#include "eig2_fixed.h"
extern "C" long t_eig(const double* g, const double* b, long n, double* l, double* v)
{
    long left = 0;
    for (long i = 0; i < n; ++i)
        if (!eig2_max_fixed(g[4 * i], g[4 * i + 1], g[4 * i + 2], g[4 * i + 3], b[i], l + i, v + 2 * i,
                            v + 2 * i + 1)) {
            l[i] = v[2 * i] = v[2 * i + 1] = NAN;
            ++left;
        }
    return left;
}
"""


@pytest.fixture(scope="module", params=[0, -3, 3])
def eig(request, tmp_path_factory):
    d = tmp_path_factory.mktemp("eig2")
    src, out = d / "t.cpp", d / "t.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off",
                    "-DNBCS_INTFP64_ESTIMATE_ULPS=(%d)" % request.param, "-I",
                    os.path.join(ROOT, "numbacs_gb300", "csrc"), str(src), "-o", str(out)],
                   check=True)
    lib = ctypes.CDLL(str(out))

    def call(g, b):
        g = np.ascontiguousarray(g)
        l, v = np.empty(len(g)), np.empty((len(g), 2))
        p = ctypes.POINTER(ctypes.c_double)
        left = lib.t_eig(g.ctypes.data_as(p), b.ctypes.data_as(p), ctypes.c_long(len(g)),
                         l.ctypes.data_as(p), v.ctypes.data_as(p))
        return l, v, left

    return call


def _gradients(kind, k, n=20000):
    rng = np.random.default_rng(k)
    f = 2.0 ** -k
    p, q, r, s = g = rng.uniform(-1, 1, (4, n)) + 1e-6
    if kind == "columns": q *= f; s *= f
    elif kind == "rows": r *= f; s *= f
    elif kind == "diagonal": q *= f; r *= f
    elif kind == "antidiagonal": p *= f; s *= f
    elif kind == "one entry": q *= f
    elif kind == "near identity": g[:] = f * g + np.array([1.0, 0.0, 0.0, 1.0])[:, None]
    elif kind == "rank one": q[:] = 4 * p * r + f * q; s[:] = 4 * r * r + f * s
    elif kind == "near rotation": s[:] = p * (1 + f * s); r[:] = -q * (1 + f * r)
    elif kind == "scales": g *= 2.0 ** rng.integers(-k - 30, 31, (4, n))
    return g.T * 2.0 ** (k % 7 * 30 - 90)


def _vector(a, d, b, m):
    e = (abs(m) + np.sqrt(m * m + 4 * b * b)) / 2
    n = np.sqrt(e * e + b * b)
    with np.errstate(invalid="ignore"):
        major, minor = np.where(n > 0, e / n, 1), np.where(n > 0, b / n, 0)
    v = np.stack([np.where(m >= 0, major, minor), np.where(m >= 0, minor, major)], -1)
    return np.where(v[:, :1] < 0, -v, v), e


@pytest.mark.parametrize("k", [0, 4, 10, 20, 30, 40, 60])
@pytest.mark.parametrize("kind", ["columns", "rows", "diagonal", "antidiagonal", "one entry",
                                  "near identity", "rank one", "near rotation", "scales"])
def test_every_component_to_its_own_last_bits(eig, kind, k):
    g = _gradients(kind, k)
    p, q, r, s = g.T
    b = p * q + r * s
    l, v, left = eig(g, b)
    P, Q, R, S = g.T.astype(np.longdouble)
    A, B, D = P * P + R * R, b.astype(np.longdouble), Q * Q + S * S
    M = (P - S) * (P + S) + (R - Q) * (R + Q)      # a - d without its cancellation
    W, e = _vector(A, D, B, M)
    use = ~np.isnan(l)
    assert left <= (len(g) if kind in ("near identity", "near rotation") and k >= 30 else 0)
    # the diagonal's difference is off by 2^-57 of the larger entry and 2^-64 of it
    # here; two roundings and the series of root and product besides
    big = np.maximum(A, D)
    tol = 2 * U + 2.0 ** -56 * big / np.maximum(abs(M) + 2 * abs(B), 1e-300)
    ok = use & (tol < 0.01)                         # (an isotropic tensor has no direction)
    assert np.all(abs(v - W)[ok] <= tol[ok, None] * abs(W)[ok] * 2)
    assert np.all(abs((v.astype(np.longdouble) ** 2).sum(1) - 1)[use] <= 3 * U)
    lam = np.minimum(A, D) + e
    assert np.all(abs(l - lam)[use] <= (1 * U + 2.0 ** -57) * 2 * lam[use])


def test_zero_off_diagonal_and_isotropic(eig):
    g = np.array([[3.0, 2.0 ** -40, -2.0 ** -40, 3.0], [1.0, -0.5, 0.5, 1.0], [0.5, -1.0, 1.0, 0.5],
                  [2.0, 1.0, 1.0, -2.0], [1.0, 1.0, 1.0, -1.5]])
    b = g[:, 0] * g[:, 1] + g[:, 2] * g[:, 3]
    l, v, left = eig(g, b)
    assert left == 0 and np.array_equal(v[:4], [[1.0, 0.0]] * 4) and np.array_equal(b[:4], [0.0] * 4)
    a, d = (g[:4, 0::2] ** 2).sum(1), (g[:4, 1::2] ** 2).sum(1)
    np.testing.assert_allclose(l[:4], np.maximum(a, d), rtol=2 * U, atol=0)
    assert v[4, 0] > 0.0 > v[4, 1]                  # the sign that leaves x positive
    # equal diagonals and an entry below the fixed point: left to the general form
    assert eig(np.array([[1.0, -1.0, 1.0, 1.0]]), np.array([2.0 ** -80]))[2] == 1
