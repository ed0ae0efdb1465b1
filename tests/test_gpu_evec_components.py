"""The smaller component of ftle_evec_2D's vectors, relative to itself: gradients
whose columns, rows or diagonals lie far apart, without cancellation in the
tensor's entries."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


@pytest.mark.parametrize("k", [0, 3, 10, 20, 30, 45, 60])
@pytest.mark.parametrize("kind", ["columns", "rows", "diagonal", "antidiagonal"])
def test_relative_error(nb, kind, k):
    rng = np.random.default_rng(k)
    n = 300
    f = 2.0 ** -k
    # one gradient [[p, q], [r, s]] a point: every third point of a (3 n, 3) map,
    # whose four neighbours are its own; positive entries, dyadic spacings
    g = rng.uniform(0.5, 1.0, (4, n)) * np.array({"columns": [1, f, 1, f], "rows": [1, 1, f, f],
                                                  "diagonal": [1, f, f, 1],
                                                  "antidiagonal": [f, 1, 1, f]}[kind])[:, None]
    if kind in ("diagonal", "antidiagonal"):
        g[0 if kind == "diagonal" else 1] *= 1.5   # the diagonal's difference does not vanish
    fm = np.zeros((3 * n, 3, 2))
    c = 3 * np.arange(n) + 1
    for at, row, half in (((c + 1, 1), 0, g[0::2]), ((c - 1, 1), 0, -g[0::2]),
                          ((c, 2), 1, g[1::2]), ((c, 0), 1, -g[1::2])):
        fm[at] = half.T
    _, v = nb.ftle_evec_2D(fm, 1.0, 1.0, 1.0)
    v = v[c, 1].astype(np.longdouble)
    p, q, r, s = g.astype(np.longdouble)   # (2 g) / (2 dx)
    a, b, d = p * p + r * r, p * q + r * s, q * q + s * s
    e = (abs(a - d) + np.sqrt((a - d) ** 2 + 4 * b * b)) / 2
    norm = np.sqrt(e * e + b * b)
    big = a >= d
    want = np.stack([np.where(big, e, b) / norm, np.where(big, b, e) / norm], -1)
    # two products and their sum (2 U each term, 1 U), the diagonal's difference
    # (4 U of its larger entry), root and normalisation (4 U)
    tol = U * (12.0 + 8.0 * np.maximum(a, d) / e)[:, None]
    assert np.all(abs(v - want) <= tol * want), (abs(v - want) / want / U).max()
