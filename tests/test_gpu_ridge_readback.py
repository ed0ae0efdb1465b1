"""The page-locked results of the ridge calls outlive the kernels that write them:
a call that raises after its launch waits before it lets go of them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["points", "fmin", "percentile", "ridges"])
def test_a_call_that_raises_has_waited(nb, name, monkeypatch):
    from numbacs_gb300.extraction import ridges as R
    rng = np.random.default_rng(2)
    f = rng.standard_normal((120, 90)) + 5.0
    a = rng.uniform(-1.5, 1.5, f.shape)
    e = np.stack([np.cos(a), np.sin(a)], -1)
    x, y = np.arange(120) * 0.5, np.arange(90) * 0.25
    call = {"points": lambda: R.ftle_ridge_pts(f, e, x, y, 0.0, 90),
            "fmin": lambda: R.ridge_pts_fmin(f, e, x, y, 0.5, 0.25, 0.0, 5.5),
            "percentile": lambda: R.percentile(f, 90.0),
            "ridges": lambda: R.ftle_ridges(f, e, x, y, 0.0, 90)}[name]
    events = []

    def check(rc):
        assert rc == 0
        events.append("launched")
        raise RuntimeError("an error that another call left behind")

    wait = R.D.synchronize
    monkeypatch.setattr(R._lib, "check", check)
    monkeypatch.setattr(R.D, "synchronize", lambda: (wait(), events.append("waited")))
    with pytest.raises(RuntimeError, match="left behind"):
        call()
    assert events == ["launched", "waited"]
