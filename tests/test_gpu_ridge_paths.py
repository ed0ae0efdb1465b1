"""Percentile selection and labelled ridges where they change form: groups of
keys around the number that is ranked by counting, ties down to the last bit,
components in shared memory and beyond it, more component sizes than the first
copy brings, warps with more ridge points than they keep."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [511, 512, 513, 514, 3000, 40000])
@pytest.mark.parametrize("q", [0.0, 10.0, 50.0, 99.9, 100.0])
def test_percentile_close_keys(nb, orc, n, q):
    from numbacs_gb300.extraction.ridges import percentile
    rng = np.random.default_rng(n)
    i = rng.permutation(n)
    close = (np.float64(0.1).view(np.int64) + i).view(np.float64)     # n neighbouring doubles
    ties = np.float64(0.1) * (1.0 + 2.0 ** -40 * (i % 3))             # three values
    two = np.where(i % 2, -close, close)
    wide = np.exp(rng.uniform(-700, 700, n)) * np.where(i % 2, 1, -1)
    for f in (close, ties, two, wide, np.full(n, 0.25), np.zeros(n), np.where(i < n // 2, 0.0, close)):
        got = percentile(f, q)
        assert got == orc.percentile(f, q), (f[:3], q)


def _expected(nb, f, e, x, y, pct, least):
    scipy_ndimage = pytest.importorskip("scipy.ndimage")
    full, mask, _, _ = nb.extraction._ftle_ridges(f, e, x, y, 0.0, pct)
    lab, n = scipy_ndimage.label(mask, np.ones((3, 3)))
    lab = lab.reshape(-1)
    idx = np.nonzero(lab)[0]
    order = idx[np.argsort(lab[idx], kind="stable")]
    counts = np.bincount(lab, minlength=n + 1)[1:]
    parts = np.split(full[order], np.cumsum(counts)[:-1]) if n else []
    return [p for p in parts if len(p) >= least], len(idx), n


@pytest.mark.parametrize("shape,smooth,pct", [((60, 50), 1, 0), ((200, 190), 1, 0),
                                              ((300, 33), 2, 50), ((700, 500), 1, 0),
                                              ((401, 600), 6, 80), ((300, 260), 1, 90),
                                              ((5, 4), 1, 0), ((3, 3), 1, 0)])
def test_labelled_ridges(nb, shape, smooth, pct):
    nx, ny = shape
    rng = np.random.default_rng(nx)
    f = rng.standard_normal((nx + smooth - 1, ny + smooth - 1))
    f = sum(f[i:i + nx, j:j + ny] for i in range(smooth) for j in range(smooth)) + 5.0
    a = rng.uniform(-1.5, 1.5, (nx, ny)) if smooth == 1 else np.full((nx, ny), 0.7)
    e = np.stack([np.cos(a), np.sin(a)], -1)
    x, y = np.arange(nx) * 0.5, np.arange(ny) * 0.25
    for least in (1, 3):
        got = nb.ftle_ridges(f, e, x, y, percentile=pct, min_ridge_pts=least)
        want, points, comps = _expected(nb, f, e, x, y, pct, least)
        assert len(got) == len(want)
        for g, w in zip(got, want):
            np.testing.assert_array_equal(g, w)
    if shape == (300, 260):
        assert points <= 8192 and comps > 1022   # the sizes come in two copies
    if shape in ((200, 190), (700, 500)):
        assert points > 8192                     # labelled on the grid


def test_ridge_points_of_every_density(nb, orc):
    rng = np.random.default_rng(9)
    x, y = np.linspace(0, 1, 333), np.linspace(0, 1, 257)
    f = np.sin(60 * x)[:, None] + 0.2 * np.cos(11 * y)[None, :] + 3.0
    e = np.zeros(f.shape + (2,))
    e[..., 0] = 1.0
    f2 = f.copy()
    f2[100:200] = rng.random((100, 257)) + 2.5
    for g in (f, f2):
        for pct in (0, 35, 97):
            np.testing.assert_array_equal(nb.ftle_ridge_pts(g, e, x, y, 0.0, pct),
                                          orc.ftle_ridge_pts(g, e, x, y, 0.0, pct))
