"""The benchmark's result line is short enough to be read back whole."""

import json

import bench


def _line():
    steps = [231.8] * 20
    return {
        "metric": bench.METRIC, "value": 25.9, "unit": "solves/s", "n_gpus": 1, "steps": 20,
        "warmup": 5, "ms_per_step": 231.9, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32+f64", "data": "synthetic",
        "config": {"workload": "w" * 300, "grid_size": 2048, "tol": 1e-6},
        "single_mixed": {"value": 21.0, "unit": "solves/s", "iterations": [100] * 6},
        "uneven_batch": {"value": 130.0, "unit": "solves/s", "problems": 96, "converged": 96,
                         "seconds": 0.7, "workload": "w" * 200},
        "adjoint": {"directions": [{"fd": 1.0, "adj": 1.0, "moved": [0, 0]}] * 64},
        "large_single": {"seconds": 0.2, "status": "converged", "stages": [["a", 1, 0.1]] * 6},
        "precision_study": {"rows": [{"Ns": 2048, "seconds_runs": [1.0, 1.0]}] * 7},
        "fp64_gpu": {"value": 13.0, "unit": "solves/s", "ratio_mixed_over_fp64": 1.9,
                     "iterations": [100] * 6},
        "iterations": [200] * 6,
        "accuracy_gate": {"pass": True, "problems": [{"backend": "fft", "status": "converged"}] * 6},
        "e2e": {"value": 25.0, "unit": "solves/s", "h2d_bytes_per_step": 1, "d2h_bytes_per_step": 1},
        "roofline": {"bound": "hbm", "achieved": 2500.0, "peak": 6551.4},
        "solve_roofline": {"achieved": 5800.0, "peak": 6551.4, "unit": "GB/s", "frac": 0.9,
                           "model": "m" * 200},
        "tangential_apply": {"f32": {"ms": 0.2}, "f64": {"ms": 0.4}},
        "gpu_launches": 1000, "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": []},
        "step_ms": {k: steps for k in ("batched", "single_mixed", "fp64_gpu", "e2e", "e2e_single")},
        "cpu_baseline": {"value": 0.007, "unit": "solves/s", "cores": 16, "kind": "port",
                         "sample": "s" * 500, "validation": {"x": [1.0] * 50}},
    }


def test_result_line_is_short_and_whole():
    line = _line()
    short, detail = bench.compact(line)
    assert len(json.dumps(short)) < 4096 < len(json.dumps(line))
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step",
                "higher_is_better", "scaling", "vs_baseline", "dtype", "data", "config", "e2e",
                "roofline", "gpu_launches", "clocks"):
        assert short[key] == line[key]
    assert short["cpu_baseline"]["value"] == 0.007 and short["accuracy_gate"] == {"pass": True}
    assert detail["adjoint"] == line["adjoint"] and detail["step_ms"] == line["step_ms"]
