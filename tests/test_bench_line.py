"""The benchmark's JSON line holds the headline keys and stays short however
large the extra sections are (no GPU)."""

import json

import bench


def test_line_is_short_and_complete():
    keep = {"metric": bench.METRIC, "value": 1.0, "unit": bench.UNIT, "n_gpus": 1, "steps": 20, "warmup": 5,
            "ms_per_step": 0.45, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
            "data": "synthetic", "config": bench.config(2048, "weno5"), "e2e": {"value": 1.0}, "gpu_launches": 300,
            "roofline": {"frac": 0.5}, "clocks": {"sm_mhz": 1965}, "parity": {"passed": True}}
    res = dict(keep, **{k: {"cases": ["x" * 1000] * 10} for k in bench.SECTIONS})
    line = bench.headline(res)
    assert json.loads(line) == keep and "\n" not in line and len(line) < 2000
