"""bench.py's printed line: one JSON object with its own figures in full, short enough
for a runner that keeps the last 30 KB of a program's output."""
import importlib.util
import json
import os

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_line_is_short_and_keeps_the_headline():
    spec = importlib.util.spec_from_file_location("bench_module", os.path.join(ROOT, "bench.py"))
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    x = 1.0 / 3.0
    row = {k: np.float64(x * 1e-7) for k in bench._LADDER_KEYS + ("rhs_evals_per_particle", "status_ok",
                                                                  "q50", "q999", "other")}
    sweep = dict({k: x * 1e5 for k in bench._SWEEP_KEYS}, cpu_baseline={"value": x, "sample": "s" * 200})
    out = {"metric": "m" * 90, "value": x * 1e8, "unit": "u", "ms_per_step": x, "steps": 20,
           "config": {"particles": 169676, "rtol": 3e-9}, "gpu_launches": 60,
           "e2e": {"value": x * 1e8, "h2d_bytes_per_step": 7416},
           "accuracy": {"bound_deg": 1.35e-4, "ladder": [row] * 42},
           "learned": {"heldout": {str(k): x for k in range(60)}},
           "c3_precision_sweep": [sweep] * 9}
    line = bench.line_of(out)
    assert "\n" not in line and len(line) < 16000
    got = json.loads(line)
    assert list(got) == list(out)
    for k in ("metric", "value", "unit", "ms_per_step", "steps", "gpu_launches"):
        assert got[k] == out[k]
    assert got["e2e"] == out["e2e"] and got["config"] == out["config"]
    assert set(got["accuracy"]["ladder"][0]) == set(bench._LADDER_KEYS)
    assert set(got["c3_precision_sweep"][0]) == set(bench._SWEEP_KEYS)
    assert out["accuracy"]["ladder"][0]["other"] == row["other"]
