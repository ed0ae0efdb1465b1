"""ftle_evec_2D's fixed-point form: gradients of any ratio and scale, tensors
that are nearly or exactly diagonal or isotropic, sizes about a block."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52


@pytest.mark.parametrize("shape", [(3, 3), (3, 131), (43, 3), (129, 65)])
@pytest.mark.parametrize("ratio", [-90, -33, -3, 0, 2, 40])
@pytest.mark.parametrize("kind", ["any", "shear", "diagonal", "rotation", "close"])
def test_against_oracle(nb, orc, shape, ratio, kind):
    nx, ny = shape
    rng = np.random.default_rng(nx + ny)
    X, Y = np.meshgrid(np.arange(nx) - 0.3 * nx, np.arange(ny) - 0.7 * ny, indexing="ij")
    noise = rng.uniform(-1, 1, (nx, ny, 2))
    A = {"any": [[1.3, -0.4], [0.7, 2.1]], "shear": [[1.0, 50.0], [1e-9, 1.0]],
         "diagonal": [[2.0, 1e-14], [-1e-14, 1.0]], "rotation": [[0.6, -0.8], [0.8, 0.6]],
         "close": [[1.0, 1e-6], [1e-6, 1.0 + 1e-6]]}[kind]
    fm = np.stack([A[0][0] * X + A[0][1] * Y, A[1][0] * X + A[1][1] * Y], -1)
    fm += noise * {"any": 0.5, "shear": 1e-3, "diagonal": 1e-10, "rotation": 1e-3,
                   "close": 1e-8}[kind]
    dx, dy = 1.0, 2.0 ** -ratio if ratio > -33 else 2.0 ** 30
    if ratio < -33:
        fm[..., 1] *= 2.0 ** -55      # one row of the gradient 2^-55 below the other
    f, v = nb.ftle_evec_2D(fm, -10.0, dx, dy)
    oev, ovec = orc.C_eig_2D(fm, dx, dy)
    l0, l1, o = oev[..., 0], oev[..., 1], ovec[..., :, 1]
    # a tensor that is off by k units of its largest entry turns the vector by
    # k EPS l1 / (l1 - l0): six roundings an entry at most in the oracle's, 2^-4
    # of one here; the normalisation adds a few
    gap = np.where(l1 > 0.0, (l1 - l0) / np.where(l1 > 0.0, l1, 1.0), 1.0)
    tol = np.minimum(EPS * (8.0 / np.maximum(gap, 1e-300) + 8.0), 2.0)[..., None]
    # (the sign of a vector along y is that of its vanishing x)
    off = np.minimum(np.abs(v - o).max(-1, keepdims=True), np.abs(v + o).max(-1, keepdims=True))
    sure = gap > 1e3 * EPS
    assert np.all(off[sure] <= tol[sure]), (off / tol)[sure].max()
    assert np.all(v[..., 0] >= 0.0)
    np.testing.assert_allclose((v ** 2).sum(-1)[l1 > 0], 1.0, rtol=0, atol=4 * EPS)
    stretched = l1 > 1.0 + 1e-6
    np.testing.assert_allclose(f[stretched], orc.ftle_from_eig(l1, -10.0)[stretched], rtol=1e-6,
                               atol=0)
    assert np.all(f[l1 < 1.0 - 1e-6] == 0.0)
