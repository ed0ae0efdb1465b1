"""Ridge calls under a limit on the polls of a grid-wide wait, run by
tests/test_gpu_ridge_give_up.py with the debug library (NBCS_LIB): at no polls all
of them raise (the asynchronous one returns NaN points), at any limit a call
raises or returns what it returns without one."""
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

import numbacs_gb300 as nb  # noqa: E402
from numbacs_gb300 import _lib, shard  # noqa: E402
from numbacs_gb300.extraction import _ftle_ridges, ftle_ridge_pts, ftle_ridges  # noqa: E402
from numbacs_gb300.extraction.ordered import ftle_ordered_ridges  # noqa: E402
from numbacs_gb300.extraction.ridges import percentile, ridge_pts_fmin  # noqa: E402


def main():
    L = _lib.load()
    assert L.nbcs_check_enabled() == 1
    nx, ny = 401, 300
    rng = np.random.default_rng(1)
    f = rng.standard_normal((nx, ny)) + 5.0
    a = rng.uniform(-1.5, 1.5, (nx, ny))
    e = np.stack([np.cos(a), np.sin(a)], -1)
    x, y = np.arange(nx) * 0.5, np.arange(ny) * 0.25
    dev = [torch.from_numpy(v).cuda() for v in (f, e, x, y)]
    ops = shard.GpuOps()
    calls = {
        "percentile": lambda: percentile(f, 90.0),
        "pts": lambda: ftle_ridge_pts(f, e, x, y, 0.0, 90),
        "pts torch": lambda: ftle_ridge_pts(*dev, 0.0, 90).cpu().numpy(),
        "pts, no percentile": lambda: ftle_ridge_pts(f, e, x, y, 0.0, 0),
        "fmin": lambda: ridge_pts_fmin(f, e, x, y, 0.5, 0.25, 0.0, 5.5),
        "ridges": lambda: np.concatenate(ftle_ridges(f, e, x, y, 0.0, 95)),
        "ordered torch": lambda: np.concatenate(
            [np.zeros((0, 2))] + ftle_ordered_ridges(*dev, 1.0, min_ridge_pts=1, percentile=99)),
        "field": lambda: _ftle_ridges(f, e, x, y, 0.0, 90)[0],
        "shard": lambda: ops.ridge_field(f, e, x, y, 0.5, 0.25, 0.0, 5.5)[1].cpu().numpy(),
    }
    want = {k: c() for k, c in calls.items()}
    given_up = finished = 0
    for polls in [0] + [1, 2, 4, 8, 16, 32, 64, 128, 256, 1024] * 8:
        _lib.check(L.nbcs_check_ridge_polls(polls))
        for name, call in calls.items():
            try:
                got = call()
            except RuntimeError as err:
                assert "did not finish" in str(err), err
                given_up += 1
                continue
            assert polls > 0, name
            assert np.array_equal(got, want[name]), (name, polls)
            finished += 1
        full, mask, _, _ = _ftle_ridges(*dev, 0.0, 90)
        full, mask = full.cpu().numpy(), mask.cpu().numpy()
        assert polls or np.isnan(full).all()
        assert (np.isnan(full).all() and mask.all()) or np.array_equal(full, want["field"])
    _lib.check(L.nbcs_check_ridge_polls(-1))
    for name, call in calls.items():
        assert np.array_equal(call(), want[name]), name
    print("gave up: all at no polls, %d in all; finished: %d" % (given_up, finished))
    assert given_up > 0


if __name__ == "__main__":
    main()
