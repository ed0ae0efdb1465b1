"""Components of up to 8192 ridge points in shapes that take many rounds of hooking:
combs whose teeth join late and level by level, hubs that come last in row-major
order, spirals, mazes; against a flood fill."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _comb(heights):
    """a tooth a column, of its own top row; neighbouring teeth meet just below the
    lower top of the two"""
    k = len(heights)
    m = np.zeros((max(heights) + 3, 2 * k), bool)
    low = [max(heights[t], heights[t + 1]) + 1 for t in range(k - 1)]
    for t in range(k):
        ends = [low[u] for u in (t - 1, t) if 0 <= u < k - 1]
        m[heights[t]:max(ends), 2 * t] = True
        if t < k - 1:
            m[low[t], 2 * t + 1] = True
    return m


def _ruler(levels, up):
    k = 1 << levels
    r = [(t & -t).bit_length() - 1 if t else levels for t in range(k)]
    return _comb([levels - v for v in r] if up else r)


def _hub(teeth, depth, rng):
    m = np.zeros((depth + 1, 2 * teeth + 1), bool)
    for t in range(teeth):
        m[rng.integers(0, depth - 1):depth, 2 * t + 1] = True
    m[depth] = True
    return m


def _spiral(n):
    m = np.zeros((n, n), bool)
    i, j, di, dj = 0, 0, 0, 1
    lo, hi = [0, 0], [n - 1, n - 1]
    while lo[0] <= hi[0] and lo[1] <= hi[1]:
        m[lo[0], lo[1]:hi[1] + 1] = True
        m[lo[0]:hi[0] + 1, hi[1]] = True
        m[hi[0], lo[1]:hi[1] + 1] = True
        m[lo[0] + 2:hi[0] + 1, lo[1]] = True
        if lo[0] + 2 <= hi[0]:
            m[lo[0] + 2, lo[1]:lo[1] + 2] = True
        lo, hi = [lo[0] + 2, lo[1] + 2], [hi[0] - 2, hi[1] - 2]
    return m


def _maze(rows, cols, rng):
    """a spanning tree of rows x cols cells"""
    m = np.zeros((2 * rows, 2 * cols), bool)
    seen, stack = {(0, 0)}, [(0, 0)]
    m[0, 0] = True
    while stack:
        i, j = stack[-1]
        ways = [(i + a, j + b) for a, b in ((0, 1), (1, 0), (0, -1), (-1, 0))
                if 0 <= i + a < rows and 0 <= j + b < cols and (i + a, j + b) not in seen]
        if not ways:
            stack.pop()
            continue
        k, l = ways[rng.integers(len(ways))]
        m[i + k, j + l] = m[2 * k, 2 * l] = True
        seen.add((k, l))
        stack.append((k, l))
    return m


def _shape(name):
    rng = np.random.default_rng(5)
    if name == "ruler up":
        return _ruler(11, True)
    if name == "ruler down":
        return _ruler(11, False)
    if name == "random comb":
        return _comb(rng.integers(0, 6, 1500).tolist())
    if name == "hub":
        return _hub(600, 20, rng)
    if name == "upside down":
        return _hub(600, 20, rng)[::-1]
    if name == "spiral":
        return _spiral(125)
    if name == "maze":
        return _maze(60, 66, rng)
    if name == "mirrored maze":
        return _maze(60, 66, rng)[::-1, ::-1]
    if name == "dots":
        return rng.random((150, 170)) < 0.3
    return rng.random((100, 100)) < 0.7


def _flood(mask):
    """components ordered by first point, points in row-major order"""
    nx, ny = mask.shape
    left, out = mask.copy(), []
    for i, j in zip(*np.nonzero(mask)):
        if not left[i, j]:
            continue
        left[i, j], todo, comp = False, [(i, j)], []
        while todo:
            a, b = todo.pop()
            comp.append((a, b))
            for c in range(max(a - 1, 0), min(a + 2, nx)):
                for d in range(max(b - 1, 0), min(b + 2, ny)):
                    if left[c, d]:
                        left[c, d] = False
                        todo.append((c, d))
        out.append(sorted(comp))
    return out


@pytest.mark.parametrize("name", ["ruler up", "ruler down", "random comb", "hub", "upside down",
                                  "spiral", "maze", "mirrored maze", "dots", "blobs"])
def test_many_rounds(nb, name):
    inner = _shape(name)
    mask = np.pad(inner, 2)
    assert mask.sum() <= 8192
    # every point above the threshold 0 is a ridge point: the direction is along the
    # level line, so that the step to the ridge is zero, and every curvature passes
    rng = np.random.default_rng(1)
    f = np.where(mask, 1.0 + 0.5 * rng.random(mask.shape), -rng.random(mask.shape))
    gx, gy = np.zeros_like(f), np.zeros_like(f)
    gx[1:-1], gy[:, 1:-1] = f[2:] - f[:-2], f[:, 2:] - f[:, :-2]
    n = np.hypot(gx, gy)
    e = np.stack([-gy, gx], -1) / np.where(n > 0, n, 1.0)[..., None]
    x, y = np.arange(mask.shape[0]) * 1.0, np.arange(mask.shape[1]) * 1.0
    got = nb.ftle_ridges(f, e, x, y, sdd_thresh=-1e300, percentile=0, min_ridge_pts=1)
    want = _flood(mask)
    assert len(got) == len(want)
    for g, w in zip(got, want):
        np.testing.assert_array_equal(np.rint(g).astype(int), w)
