"""ftle_evec_2D and the batch's FTLE give a point the same bits whatever lies
beside it: in a block of rows, next to particles that did not move or left the
number range, and in a batch as in a single call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _map(nx, ny, seed=3):
    rng = np.random.default_rng(seed)
    x, y = np.linspace(0.0, 2.0, nx), np.linspace(0.0, 1.0, ny)
    X, Y = np.meshgrid(x, y, indexing="ij")
    for _ in range(3):
        a, b, c, d = rng.uniform(0.15, 0.4, 2).tolist() + rng.uniform(0.0, 6.0, 2).tolist()
        X = X + a * np.sin(np.pi * Y + c)
        Y = Y + b * np.sin(np.pi * X + d)
    return np.stack([X, Y], -1), x, y


def _holes(fm, kind):
    """the map with patches and single points that need the general form"""
    nx, ny = fm.shape[:2]
    rng = np.random.default_rng(nx)
    if kind == "still":
        fm[nx // 3:nx // 2, ny // 4:ny // 2] = fm[nx // 3, ny // 4]
    i, j = rng.integers(0, nx, 40), rng.integers(0, ny, 40)
    fm[i, j] = {"still": fm[0, 0], "nan": np.nan, "inf": np.inf, "far": 2.0 ** 80}[kind]
    return fm


@pytest.mark.parametrize("kind", ["still", "nan", "inf", "far"])
@pytest.mark.parametrize("ny", [33, 64, 131])
def test_row_blocks_give_the_whole_fields_bits(nb, kind, ny):
    fm, x, y = _map(90, ny)
    fm = _holes(fm, kind)
    dx, dy = x[1] - x[0], y[1] - y[0]
    f, v = nb.ftle_evec_2D(fm, -4.0, dx, dy)
    for e0, e1 in ((0, 31), (1, 40), (29, 62), (50, 90)):
        g, w = nb.ftle_evec_2D(np.ascontiguousarray(fm[e0:e1]), -4.0, dx, dy)
        np.testing.assert_array_equal(g[1:-1], f[e0 + 1:e1 - 1])
        np.testing.assert_array_equal(w[1:-1], v[e0 + 1:e1 - 1])


def test_sharded_ridges_with_still_water(nb):
    """three emulated ranks in turn on one GPU, a flow that leaves the particles
    outside the velocity box where they are: FTLE, directions and ridge points of
    the single-GPU pipeline"""
    from numbacs_gb300 import shard
    t, a = np.linspace(0.0, 10.0, 9), np.linspace(0.0, 1.0, 17)
    X, Y = np.meshgrid(a, a, indexing="ij")
    U = np.broadcast_to(np.sin(3 * X) * np.cos(5 * Y), (9, 17, 17)) + 0.1 * t[:, None, None]
    V = np.broadcast_to(np.cos(4 * X) * np.sin(6 * Y), (9, 17, 17)) - 0.05 * t[:, None, None]
    flow = nb.get_flow_2D(*nb.get_interp_arrays_2D(t, a, a, U.copy(), V.copy()))
    x, y, p = np.linspace(-0.3, 1.3, 121), np.linspace(-0.25, 1.2, 77), np.array([1.0])
    fm = nb.flowmap_grid_2D(flow, 0.0, 6.0, x, y, p)
    assert np.array_equal(fm[0, 0], [x[0], y[0]])
    f, v = nb.ftle_evec_2D(fm, 6.0, x[1] - x[0], y[1] - y[0])
    ops, states, rows = shard.GpuOps(), [], []
    for r in range(3):
        st, owned = shard.block_ftle(ops, r, 3, flow, 0.0, 6.0, x, y, p)
        i0, i1, e0, _ = st["rows"]
        np.testing.assert_array_equal(ops.to_numpy(st["ev"])[i0 - e0:i1 - e0], v[i0:i1])
        states.append(st)
        rows.append(owned)
    np.testing.assert_array_equal(np.concatenate(rows), f)
    pts = np.concatenate([shard.block_ridge_pts(ops, st, f, 0.0, 80) for st in states])
    assert len(pts) > 0
    np.testing.assert_array_equal(pts, nb.ftle_ridge_pts(f, v, x, y, 0.0, 80))


@pytest.mark.parametrize("h", [2.0 ** -35, 2.0 ** -34, 2.0 ** -33, 2.0 ** -32, 2.0 ** -20, 2.0 ** -3])
def test_batch_matches_the_single_call_at_any_spacing(nb, h):
    from numbacs_gb300.batch import Field, FTLEBatch
    dg, p, _ = nb.get_predefined_flow("double_gyre", int_direction=-1.0)
    x, y = 0.5 + h * np.arange(40), 0.375 + h * np.arange(37)
    b = FTLEBatch([Field(dg, 0.0, -6.0, x, y, p)], precision="fp64", blocks_per_sm=2, graph=False)
    b.run()
    fm, f, v, _ = [a.cpu().numpy() for a in b.results()[0]]
    g, w = nb.ftle_evec_2D(fm, -6.0, x[1] - x[0], y[1] - y[0])
    np.testing.assert_array_equal(g, f)
    np.testing.assert_array_equal(w, v)
