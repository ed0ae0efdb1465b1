"""FP64 integrator where its arithmetic or its kernel changes form: grids around
the size up to which products stay on the FP64 pipe, arguments beyond the
integer sine's range, coefficients and weights of zero, values that the integer
products do not take, particles outside and on the edges of the box."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1), (95, 97), (100, 96), (101, 97)])
@pytest.mark.parametrize("t0", [0.0, 300.0])
def test_double_gyre_sizes(nb, orc, shape, t0):
    x, y = np.linspace(0, 2, shape[0]), np.linspace(0, 1, shape[1])
    fl, p, _ = nb.get_predefined_flow("double_gyre", int_direction=-1.0)
    fm, st = nb.flowmap_grid_2D(fl, t0, -10.0, x, y, p, return_stats=True)
    ofm, _, ost = orc.flowmap_grid_2D(orc.double_gyre(), t0, -10.0, x, y, p, return_status=True)
    # the sines differ from libm's in the last bit only: the bar of the parity tests
    err = np.abs(fm - ofm).max(axis=-1)
    assert np.all(st == ost, axis=-1).mean() >= 0.999
    assert err.max() <= 2e-6 and np.median(err) <= 2e-12


def _flow(nb, orc, U, V, **kw):
    t, x, y = 3.0 * np.arange(U.shape[0]), np.linspace(-20, 20, U.shape[1]), np.linspace(
        0, 30, U.shape[2])
    grid, cu, cv = nb.get_interp_arrays_2D(t, x, y, U, V)
    og, ocu, ocv = orc.get_interp_arrays_2D(t, x, y, U, V)
    return nb.get_flow_2D(grid, cu, cv, **kw), orc.spline_flow(og, ocu, ocv, **kw)


def _same(nb, orc, fl, ofl, x, y, t0=24.0, T=-18.0, rtol=1e-6, atol=1e-8):
    p = np.array([-1.0])
    fm, status, st = nb.flowmap_grid_2D(fl, t0, T, x, y, p, rtol=rtol, atol=atol,
                                        return_status=True, return_stats=True)
    ofm, ostatus, ost = orc.flowmap_grid_2D(ofl, t0, T, x, y, p, rtol=rtol, atol=atol,
                                            return_status=True)
    np.testing.assert_array_equal(status, ostatus)
    np.testing.assert_array_equal(st, ost)
    np.testing.assert_array_equal(fm, ofm)


@pytest.mark.parametrize("spherical", [0, 1])
@pytest.mark.parametrize("case", ["plain", "land", "one", "tiny", "huge", "still"])
def test_spline_values(nb, orc, spherical, case):
    T3, X3, Y3 = np.meshgrid(3.0 * np.arange(9), np.linspace(-20, 20, 11), np.linspace(0, 30, 9),
                             indexing="ij")
    k = 1.0 if spherical else 1.0 / 111.0
    U = k * 30.0 * np.sin(0.15 * X3 + 0.05 * T3) * np.cos(0.1 * Y3)
    V = k * 20.0 * np.cos(0.12 * X3) * np.sin(0.2 * Y3 - 0.03 * T3)
    if case == "land":
        U[:, 6:], V[:, 6:] = 0.0, 0.0
    elif case == "one":
        V[:] = 0.0
    elif case == "tiny":
        U, V = U * 1e-90, V * 1e-200
    elif case == "huge":
        V = V * 1e-3
        U[:, :, 7:] *= 1e3
    elif case == "still":
        U[:], V[:] = 0.0, 0.0
    fl, ofl = _flow(nb, orc, U, V, spherical=spherical)
    # on the nodes, off them, on the edges and outside the box
    x = np.concatenate([np.linspace(-20, 20, 11), [-20 - 1e-12, 20 + 1e-12, 3.3, 19.9, 25.0]])
    y = np.concatenate([np.linspace(0, 30, 9), [-1e-13, 30 + 1e-12, 7.7, 45.0]])
    _same(nb, orc, fl, ofl, x, y)


def test_high_latitudes(nb, orc):
    """above 45 degrees the metric takes the sine series"""
    t, x, y = 3.0 * np.arange(9), np.linspace(-20, 20, 11), np.linspace(30, 80, 9)
    T3, X3, Y3 = np.meshgrid(t, x, y, indexing="ij")
    U, V = 20.0 * np.sin(0.15 * X3 + 0.05 * T3), 15.0 * np.cos(0.12 * X3 + 0.1 * Y3)
    grid, cu, cv = nb.get_interp_arrays_2D(t, x, y, U, V)
    og, ocu, ocv = orc.get_interp_arrays_2D(t, x, y, U, V)
    _same(nb, orc, nb.get_flow_2D(grid, cu, cv, spherical=1),
          orc.spline_flow(og, ocu, ocv, spherical=1), np.linspace(-18, 18, 21),
          np.linspace(32, 78, 23))
