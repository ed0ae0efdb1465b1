"""Start and end times that are NaN or infinite, in either direction: the statuses
of the oracle, from the single call, the point list and the batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAN, INF = float("nan"), float("inf")


@pytest.mark.parametrize("t0,T", [(NAN, 2.0), (NAN, -2.0), (0.0, NAN), (1.0, NAN), (NAN, NAN),
                                  (INF, 2.0), (-INF, 2.0), (INF, -INF), (-1e300, 2.0), (0.0, 2.0)])
@pytest.mark.parametrize("direction", [1.0, -1.0])
@pytest.mark.parametrize("kind", ["double_gyre", "bickley_jet", "spline"])
def test_statuses(nb, orc, kind, direction, t0, T):
    from numbacs_gb300.batch import Field, FTLEBatch
    x, y = np.linspace(0.1, 0.9, 5), np.linspace(0.2, 0.7, 3)
    if kind == "spline":
        t, a = np.linspace(-4.0, 4.0, 9), np.linspace(0.0, 1.0, 9)
        T3, X3, Y3 = np.meshgrid(t, a, a, indexing="ij")
        U, V = np.sin(3 * X3 + T3) * 0.1, np.cos(2 * Y3 - T3) * 0.1
        flow = nb.get_flow_2D(*nb.get_interp_arrays_2D(t, a, a, U, V))
        oflow = orc.spline_flow(*orc.get_interp_arrays_2D(t, a, a, U, V))
        p = np.array([direction])
    else:
        flow, p, _ = nb.get_predefined_flow(kind)
        p = p.copy()
        p[0] = direction
        oflow = getattr(orc, kind)()
    _, want, _ = orc.flowmap_grid_2D(oflow, t0, T, x, y, p, nmax=60, return_status=True)
    _, st = nb.flowmap_grid_2D(flow, t0, T, x, y, p, max_steps=60, return_status=True)
    assert np.array_equal(st, want), (st, want)
    pts = np.stack([v.ravel() for v in np.meshgrid(x, y, indexing="ij")], -1)
    _, sp = nb.flowmap(flow, t0, T, pts, p, max_steps=60, return_status=True)
    assert np.array_equal(sp.reshape(want.shape), want)
    b = FTLEBatch([Field(flow, t0, T, x, y, p)], precision="fp64", blocks_per_sm=2, graph=False,
                  max_steps=60)
    b.run()
    assert np.array_equal(b.results()[0][3].cpu().numpy(), want)
