"""FTLE and Cauchy-Green kernels where their integer arithmetic changes form:
differences and spacings at the edges of its range, zeros, infinities, NaN,
and rows that end inside a warp."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _map(nx, ny, seed=0):
    rng = np.random.default_rng(seed)
    X, Y = np.meshgrid(np.linspace(0, 2, nx), np.linspace(0, 1, ny), indexing="ij")
    fm = np.stack([X + 0.3 * np.sin(7 * Y + 3 * X), Y + 0.2 * np.cos(5 * X)], -1)
    return fm + 1e-3 * rng.standard_normal(fm.shape)


def _check(nb, orc, fm, dx, dy):
    with np.errstate(all="ignore"):
        ev, vec = nb.C_eig_2D(fm, dx, dy)
        oev, ovec = orc.C_eig_2D(fm, dx, dy)
        np.testing.assert_array_equal(ev, oev)
        np.testing.assert_array_equal(vec, ovec)
        # two logarithms within 0.55 and 1 ulp, and a product each: 2.3 ulp
        np.testing.assert_allclose(nb.ftle_grid_2D(fm, -10.0, dx, dy),
                                   orc.ftle_grid_2D(fm, -10.0, dx, dy), rtol=6e-16, atol=0)
        np.testing.assert_allclose(nb.ftle_from_eig(oev[..., 1].copy(), -10.0),
                                   orc.ftle_from_eig(oev[..., 1], -10.0), rtol=6e-16, atol=0)


@pytest.mark.parametrize("k", [-1000, -300, -64, -40, 0, 40, 66, 130, 300, 500])
@pytest.mark.parametrize("j", [-33, 0, 33])
def test_scaled_maps(nb, orc, k, j):
    fm = np.ldexp(_map(37, 29), k)
    _check(nb, orc, fm, np.ldexp(0.3, j), np.ldexp(0.7, j))


@pytest.mark.parametrize("shape", [(3, 3), (3, 200), (33, 31), (65, 129)])
def test_zeros_infinities_nan(nb, orc, shape):
    nx, ny = shape
    rng = np.random.default_rng(3)
    for special in (0.0, np.inf, -np.inf, np.nan, 1e200, 1e-200):
        fm = _map(nx, ny, 1)
        fm[rng.random(fm.shape) < 0.05] = special
        _check(nb, orc, fm, 0.01, 0.02)
    X, Y = np.meshgrid(np.arange(nx, dtype=float), np.arange(ny, dtype=float), indexing="ij")
    for fm in (np.stack([X, Y], -1), np.stack([X + 0.5 * Y, Y], -1), np.stack([Y, -X], -1),
               np.zeros((nx, ny, 2)), np.stack([2.0 * X, Y], -1)):
        _check(nb, orc, fm, 1.0, 1.0)


def test_fused_entry_point_on_zero_gradients(nb, orc):
    X, Y = np.meshgrid(np.arange(40.0), np.arange(50.0), indexing="ij")
    for fm in (np.stack([X + 0.5 * Y, Y], -1), np.stack([3.0 * X, 0.25 * Y], -1)):
        f, v = nb.ftle_evec_2D(fm, -10.0, 1.0, 1.0)
        oev, ovec = orc.C_eig_2D(fm, 1.0, 1.0)
        # the mantissa's log is FP32 (3e-7), the vector a few ulp
        np.testing.assert_allclose(f, orc.ftle_from_eig(oev[..., 1], -10.0), rtol=1e-6, atol=0)
        np.testing.assert_allclose(v, ovec[..., :, 1], rtol=0, atol=1e-15)
