"""The bench line stays short: what explains its figures goes to stderr."""
from __future__ import annotations

import json

import bench

V, E = 16777216, 504997749

# As large as the headline run makes it.
LINE = {
    "metric": bench.METRIC, "value": 1392.83, "unit": "GB/s", "n_gpus": 1, "steps": 20, "warmup": 5,
    "ms_per_step": 60.6041, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
    "dtype": "f32 (f64 residual and dangling mass)",
    "data": "synthetic R-MAT (stands in for Graph500/GraphChallenge inputs)",
    "config": bench.workload_config(24, V, E, 503316, 1), "iterations_per_step": 38, "converged": True,
    "graph_preparation_s": 14.19, "gpu_launches": 123456,
    "roofline": {"kernel": "pr_rows + pr_chunks", "bound": "hbm", "achieved": 1434.2, "peak": 6545.4,
                 "peak_kind": "measured HBM copy (MEASURED_PEAKS.json)", "unit": "GB/s", "frac": 0.2191,
                 "frac_of_8tbs_spec": 0.1793, "traffic": 2729000000, "traffic_is": "x" * 80,
                 "algorithmic_bytes_per_launch": 2221317592, "ms_per_working_launch": 1.54873,
                 "kernel_ms_per_step": {"pr_rows": 12.3456, "pr_chunks": 45.6789}, "launches_per_step": 40,
                 "working_launches_per_step": 38, "share_of_step": 0.9712},
    "e2e": {"value": 608.31, "unit": "GB/s", "h2d_bytes_per_step": 2087099864, "d2h_bytes_per_step": 67108864,
            "what": "x" * 150, "ms_per_step": 138.76, "breakdown": {"kernel_ms": {str(k): 1.234 for k in range(12)}}},
    "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": ["sw_power_cap"], "samples": 11},
    "kernel_ms_per_step": {f"kernel_{k}": 1.2345 for k in range(8)},
    "accuracy": {"l1_error_vs_fp64_oracle": 6.612345678901234e-08, "linf_error_vs_fp64_oracle": 5.012345678901234e-11,
                 "oracle": "x" * 70, "target_l1": 1e-6},
    "cpu_baseline": {"value": 18.612, "unit": "GB/s", "cores": 16, "kind": "port", "sample": "x" * 120},
    "algorithms": {"rmat24": {"runs_ms": [1.0] * 500}}, "harness": [{"dataset": "rmat24", "runs": [0.1] * 500}],
}


def leaves(x, path=()):
    if isinstance(x, dict) and x:
        return {k: v for key, y in x.items() for k, v in leaves(y, path + (key,)).items()}
    return {path: x}


def test_the_line_is_short_and_nothing_is_lost():
    before = json.dumps(LINE)
    line, details = bench.split_details(LINE)
    assert json.dumps(LINE) == before
    assert len(json.dumps(line)) < 2400
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
                "vs_baseline", "dtype", "data", "config", "clocks", "gpu_launches", "roofline", "cpu_baseline", "accuracy"):
        assert key in line
    assert set(line["e2e"]) >= {"value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"}
    a, b = leaves(line), leaves(details)
    assert not set(a) & set(b) and {**a, **b} == leaves(LINE)


def test_a_line_without_details():
    line = {"metric": "m", "value": 1.0, "e2e": {"value": 1.0}}
    assert bench.split_details(line) == (line, {})
