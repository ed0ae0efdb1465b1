"""Spline prefilter where its chunks, tiles and integer arithmetic end: axis
lengths around the chunk of eight and the shared-memory tile, and values that
the integer arithmetic does not take.  Bit for bit the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _both(nb, orc, u, v):
    t, x, y = (np.arange(float(n)) for n in u.shape)
    _, cu, cv = nb.get_interp_arrays_2D(t, x, y, u, v)
    with np.errstate(all="ignore"):
        np.testing.assert_array_equal(cu, orc.prefilter_3d(u))
        np.testing.assert_array_equal(cv, orc.prefilter_3d(v))


@pytest.mark.parametrize("n", [2, 3, 4, 9, 10, 11, 12, 17, 18, 19, 26, 33])
def test_axis_lengths(nb, orc, n):
    rng = np.random.default_rng(n)
    for shape in ((n, 3, 5), (5, n, 33), (3, 4, n)):
        _both(nb, orc, rng.standard_normal(shape), rng.standard_normal(shape))


@pytest.mark.parametrize("ny", [379, 380, 381, 700])
def test_tile_limit(nb, orc, ny):
    rng = np.random.default_rng(ny)
    _both(nb, orc, rng.standard_normal((2, 35, ny)), rng.standard_normal((2, 35, ny)))


@pytest.mark.parametrize("special", [0.0, 1e-310, 1e-100, 1e150, np.inf, np.nan])
def test_values(nb, orc, special):
    rng = np.random.default_rng(1)
    u, v = rng.standard_normal((2, 21, 14, 30))
    u[rng.random(u.shape) < 0.02] = special
    v[:] = special
    v[3:9] = 2.0
    _both(nb, orc, u, v)
