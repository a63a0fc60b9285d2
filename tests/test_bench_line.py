"""The default run's line on standard output stays short however long the whole
record is, and keeps every field that the record's readers take from it (no
GPU)."""
import json
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)


@pytest.fixture(scope="module")
def bench():
    argv = sys.argv
    sys.argv = ["bench.py"]
    try:
        import bench as b
        yield b
    finally:
        sys.argv = argv


def _record(bench, cpu=True):
    args = bench.parse()
    form = {"stage_ms": dict.fromkeys(bench.STAGES, 1.0 / 3), "ms_per_step": 29.123456789012345,
            "per_step": dict.fromkeys(["contacts", "meetings", "new_keys", "checks", "cross_checks", "border_objects",
                                       "buckets", "expired", "candidates"], 123456789.123),
            "value": 3.3333333333e8, "meetings_per_step": list(range(2000))}
    lat = {"p50_ms": 1.0 / 3, "p99_ms": 2.0 / 3, "queries": 1200, "finished": 1200, "qps": 200.1, "rate_req_s": 200.0,
           "rates": {str(k): {"p50_ms": 0.1} for k in range(100)}, "two_hop_1k_seeds": {"p50_ms": 0.5, "p99_ms": 0.7,
                                                                                      "mean_reached": 3e5}}
    parity = {k: {"steps": 25, "meetings": 123456789, "mismatching_steps": list(range(1000)), "compared": "x" * 300}
              for k in ("tuned_vs_plain", "oracle")}
    return {"metric": bench.METRIC, "value": 3.4e8, "unit": bench.UNIT, "n_gpus": 1, "steps": 20, "warmup": 5,
            "ms_per_step": 29.1, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic", "config": bench.workload_config(args, 10_000_000, "tuned"),
            "roofline": bench.roofline(form, 10_000_000, 1 << 30, "tuned"),
            "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": [], "samples": 8},
            "e2e": {"value": 2.68276002e8, "unit": bench.UNIT, "h2d_bytes_per_step": 160000000,
                    "d2h_bytes_per_step": 201235604, "steps": 20},
            "cpu_baseline": {"value": 3.0e6, "unit": bench.UNIT, "cores": 16, "kind": "port", "sample": "y" * 300,
                             "ms_per_step": 3294.0167039999997, "steps": 3, "same_config": True,
                             "cpu_model": "z"} if cpu else None,
            "parity": parity, "gpu_launches": 1234, "serving": lat if cpu else None,
            "compaction": {"source_keys": 1 << 30, "ms": 12.3, "source_keys_per_s": 5e9, "note": "n" * 500,
                           "serving": lat},
            "forms": {k: dict(form) for k in ("tuned", "plain", "batch64", "skew50m")}, "parity_ok": False}


@pytest.mark.parametrize("cpu", [True, False])
def test_line_is_short_and_whole(bench, cpu):
    rec = _record(bench, cpu)
    assert len(json.dumps(rec)) > 20_000
    text = json.dumps(bench.short_line(rec))
    assert len(text) < 4000 and "\n" not in text
    line = json.loads(text)
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
              "vs_baseline", "dtype", "data", "config", "clocks", "e2e", "gpu_launches", "parity_ok"):
        assert line[k] == rec[k], k
    for k in ("achieved", "peak", "unit", "frac", "traffic", "algorithmic_bytes"):
        assert line["roofline"][k] == rec["roofline"][k]
    if cpu:
        assert line["cpu_baseline"]["value"] == rec["cpu_baseline"]["value"]
        assert line["serving"]["two_hop_1k_seeds"] == {"p50_ms": 0.5, "p99_ms": 0.7}
    assert line["parity"]["oracle"]["mismatching_steps"] == list(range(16))
    assert set(line["forms"]) == {"tuned", "plain", "batch64", "skew50m"}
