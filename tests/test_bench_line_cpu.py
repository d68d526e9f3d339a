"""bench.py's result is one short line on standard output, whatever the blocks
hold: records of a run keep the last 3,000 characters of it."""
from __future__ import annotations

import importlib.util
import json
import sys

from conftest import ROOT


def load():
    spec = importlib.util.spec_from_file_location("bench_module", ROOT / "bench.py")
    mod = importlib.util.module_from_spec(spec)
    sys.modules["bench_module"] = mod
    spec.loader.exec_module(mod)
    return mod


def test_line_stays_short(capsys):
    x = 123456789.123456789
    third = 0.1234567890123456
    line = {
        "metric": "body-steps/s", "value": x, "unit": "body-steps/s", "n_gpus": 1, "steps": 20, "warmup": 5,
        "ms_per_step": third, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
        "data": "synthetic " + "x" * 100,
        "config": {"workload": "w" * 110, "bodies": 300149, "theta": 1.05, "dt_days": third, "mode": "fp64_list",
                   "seed": 2, "outer": 0.1, "trojan": 0.0, "l2": "l" * 50, "parallelism": "replicas x1"},
        "roofline": {"kernel": "k" * 60, "bound": "fp64", "achieved": third, "peak": third, "unit": "TFLOP/s",
                     "frac": third, "peak_source": "p" * 70, "work": "w" * 60, "traffic": 123456789,
                     "traffic_unit": "bytes per launch (ncu)", "hbm_view": {"gbs": x, "frac": third, "peak": x}},
        "phases_ms_per_step": {k: third for k in ("kick_drift_bbox", "keys", "sort", "permute", "build", "forces")},
        "interactions_per_body": x, "interactions_per_s": x,
        "accuracy": {"median_rel_err": third, "p99_rel_err": third, "sample": 4096, "against": "FP64 direct sum"},
        "e2e": {"value": x, "unit": "body-steps/s", "h2d_bytes_per_step": 26413112, "d2h_bytes_per_step": 26413112},
        "gpu_launches": 640,
        "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": ["none"], "samples": 10, "power_w": x},
        "cpu_baseline": {"value": x, "unit": "body-steps/s", "cores": 16, "kind": "port", "sample": "s" * 90},
    }
    blocks = {"forms_4m": {"rows": [third] * 5000}, "csv_ingest": None}
    load().print_result(line, blocks)
    out, err = capsys.readouterr()
    assert out.count("\n") == 1 and len(out) < 2900
    got = json.loads(out)
    assert set(got) == set(line) and got["value"] == x and got["ms_per_step"] == third
    assert got["e2e"]["h2d_bytes_per_step"] == 26413112 and abs(got["e2e"]["value"] / x - 1) < 1e-5
    assert json.loads(err) == {"forms_4m": blocks["forms_4m"]}
