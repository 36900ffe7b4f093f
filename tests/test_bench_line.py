"""bench.py's line on stdout: the contract's keys, short enough for a log that keeps its last 1500 characters."""
import json

import bench


def test_headline_is_complete_and_short():
    x = 1234.5678901234567
    leg = {"jobs": 8, "fit_ms_p50": x, "fit_ms_p99": x, "phase_ms_p50": {str(i): x for i in range(60)}}
    line = {
        "metric": bench.METRIC, "value": x, "unit": bench.UNIT, "n_gpus": 8, "steps": 200, "warmup": 10, "ms_per_step": x,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f" * 96, "data": "s" * 60,
        "config": bench.workload_config(), "run": {"launch": "l" * 400},
        "fp64": {"value": x, "unit": "evals/s", "ms_per_step": x, "kernel_ms": x, "traffic": x},
        "mixed_over_fp64": x, "accuracy": {"abs_dnll_mixed_vs_fp64": x, "grad_rel_err_mixed_vs_fp64": x},
        "clocks": {"sm_mhz": 1953.5, "sm_max_mhz": 1965.0, "reasons": ["sw_power_cap"], "samples": 6, "power_w_max": x},
        "e2e": {"value": x, "unit": bench.UNIT, "h2d_bytes_per_step": 184, "d2h_bytes_per_step": 192, "ms_per_step": x},
        "gpu_launches": 600,
        "roofline": {"bound": "hbm", "achieved": x, "peak": 6650.0, "unit": "GB/s", "frac": x, "kernel_ms": x, "kernel": "k"},
        "hessian": {"n_params": 23, "exact_ms": x}, "gram": {"ms": x},
        "toy_fit": {"sweep": [{"rate_per_s": r, "mixed": leg, "fp64": leg} for r in (1.0, 50.0)]},
        "cpu_baseline": {"sample": "s" * 300},
    }
    text = json.dumps(bench.headline(line))
    assert len(text) < 1400
    out = json.loads(text)
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
                "vs_baseline", "dtype", "data", "config", "clocks", "e2e", "gpu_launches"):
        assert key in out, key
    for key in ("value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"):
        assert key in out["e2e"]
    for key in ("sm_mhz", "sm_max_mhz", "reasons"):
        assert key in out["clocks"]
    assert abs(out["value"] / x - 1) < 1e-6
