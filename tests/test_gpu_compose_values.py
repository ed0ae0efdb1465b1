"""Flow-map composition where its integer arithmetic changes form: differences
across zero and across powers of two, constant and unusual values, points on the
edges of the box and outside it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nT", [1, 2, 5])
@pytest.mark.parametrize("special", [None, 0.0, np.inf, np.nan, 1e-300, 3.0, 2.0])
def test_compose_values(nb, orc, nT, special):
    nx, ny = 37, 26
    rng = np.random.default_rng(4)
    X, Y = np.meshgrid(np.linspace(-3.0, 5.0, nx), np.linspace(-1.0, 4.0, ny), indexing="ij")
    maps = np.stack([np.stack([X + 0.4 * np.sin(Y + k), Y + 0.3 * np.cos(X - k)], -1)
                     for k in range(nT)])
    maps[:, 5:9, 3:9] = [-3.0, 4.0]                # a corner of the box
    maps[:, 20, :, 0] = 5.0                        # its far edge
    maps[:, 21, :, 0] = np.nextafter(5.0, 6.0)     # and beyond it
    maps[:, :, 11, 1] = -1.0
    if special is not None:
        maps[rng.random(maps.shape) < 0.03] = special
    grid = nb.UCGrid((-3.0, 5.0, nx), (-1.0, 4.0, ny))
    got = nb.flowmap_composition(maps, grid, nT)
    want = orc.flowmap_composition(maps, grid, nT)
    np.testing.assert_array_equal(got, want)
