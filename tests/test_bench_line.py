"""bench.py's result line on the CPU: short enough to be read whole, with every
key that a reader of it needs."""
import json
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

x = 123456789.12345679


def test_result_line_is_short_and_complete():
    import bench
    full = {
        "metric": bench.METRIC, "value": x, "unit": bench.UNIT, "n_gpus": 1, "steps": 20, "warmup": 5, "ms_per_step": x,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic: " + "d" * 60,
        "config": bench.workload_config(1 << 22, ("learned", 0.045868172414943065, 0.0), "hernquist"),
        "e2e": {"value": x, "unit": bench.UNIT, "h2d_bytes_per_step": 1 << 28, "d2h_bytes_per_step": 1 << 28, "calls": "c" * 200},
        "gpu_launches": 123456,
        "roofline": {"bound": "fp32", "achieved": x, "peak": x, "unit": "TFLOP/s", "frac": x, "traffic": 1 << 30, "kernel": "k" * 50},
        "headline": {"rms": x, "p99": x, "target_rms": x, "guard": {"checks": 1}, "build_ms": x, "walk_ms": x},
        "ratios": {"learned_vs_fixed_theta_equal_rms": x, "error_rule_vs_fixed_theta_equal_rms": x},
        "comparisons": {"c" * 10: "c" * 3000}, "calibration": {"c": [x] * 500}, "walk_stats": {"mask_hist": [0] * 33},
        "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": ["sw_power_cap", "hw_slowdown"], "samples": 100},
        "cpu_baseline": {"value": x, "unit": bench.UNIT, "cores": 1, "kind": "port", "sample": "s" * 400},
        "workloads": {name: {"value": x, "clocks": {}, "unit": "u" * 20} for name, _, _ in bench.COMPANIONS},
    }
    full["workloads"]["galaxy"] = {"error": "timed out"}
    line = bench.result_line(full)
    assert "\n" not in line and len(line.encode()) <= 1500, len(line)
    got = json.loads(line)
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
                "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "clocks"):
        assert key in got
    for key in ("metric", "value", "ms_per_step", "config", "clocks"):
        assert got[key] == full[key]
    assert set(got["e2e"]) == {"value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"}
    assert got["workloads"]["galaxy"] is None and got["workloads"]["hernquist"] > 0
