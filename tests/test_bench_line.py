"""bench.py's line: one JSON object with the headline whole, short enough for a
reader of the output's last few thousand characters; the blocks in full go to
standard error."""
import importlib
import json

bench = importlib.import_module("bench")


def record():
    long = "a description of what was measured and how, of a hundred characters and more, as the blocks hold " * 3
    roof = {"bound": "hbm", "achieved": 1.0, "peak": 2.0, "unit": "GB/s", "frac": 0.5, "traffic": 1e11, "kernel": "k",
            "peak_source": long, "alg_bytes_per_state": 8.0, "eval_ms_per_step": 3.0, "eval_launches": 20,
            "fp64": {"achieved": 1.0, "peak": 2.0, "unit": "TFLOP/s", "frac": 0.5, "pipe_frac": 0.6, "source": long}}
    cpu = {"value": 2e5, "unit": "Jacobians/s", "cores": 16, "kind": "port", "sample": long}
    parity = {"states": 700, "rates_max_rel": 1e-12, "rates_pass": True, "jacobian_pass": True, "rates_bar": long}
    curve = [{"tol": t, "ms": 1.0, "fallback_frac": 0.123456789, "speedup_vs_fp64": 1.23456789} for t in
             (1.0, 0.5, 0.3, 0.1, 0.01, 0.001)]
    step = {"kernel": long, "ms": 123.456789, "states_per_s": 1e7}
    return {"metric": bench.METRIC, "value": 1.7e7, "unit": "Jacobians/s", "n_gpus": 1, "steps": 20, "warmup": 5,
            "ms_per_step": 60.7, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic", "config": {"workload": "w", "l2": long[:120]}, "roofline": roof, "cpu_baseline": cpu,
            "e2e": {"value": 7e6, "unit": "Jacobians/s", "h2d_bytes_per_step": 1, "d2h_bytes_per_step": 2, "steps": 5,
                    "call_ms": [150.0] * 5, "median_call_ms": 150.0, "path": long,
                    "link": {"d2h_gbs": 170.0, "d2h_floor_ms_per_step": 143.0, "what": long}},
            "gpu_launches": 40, "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": []}, "parity": parity,
            "configs": {"config_%d" % i: {"value": 1.234567891e7, "unit": "states/s", "workload": long,
                                          "roofline": roof, "cpu_baseline": cpu, "parity": parity} for i in range(7)},
            "surrogate": {"network_speedup_vs_fp64": 9.1, "err_median": 0.12, "with_fallback": curve, "note": long},
            "implicit_step": {"states": 1, "h": long, "synthetic500": {"factor": step},
                              **{k: step for k in ("factor", "solve", "ros2_step", "ros2_step_sparse")}}}


def test_line_is_short_and_whole():
    rec = record()
    line, detail = bench.split_record(rec)
    text = json.dumps(line)
    assert "\n" not in text and len(text) < 3500
    required = ["metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
                "vs_baseline", "dtype", "data", "config", "gpu_launches", "clocks"]
    assert all(line[k] == rec[k] for k in required)
    for k in ("value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"):
        assert line["e2e"][k] == rec["e2e"][k]
    assert line["configs"]["config_3"] == {"value": 1.234567891e7, "unit": "states/s"}
    assert line["surrogate"]["speedup_at_tol"]["0.001"] == 1.235
    assert line["implicit_step_ms"]["ros2_step"] == 123.456789
    assert all(detail[k] == rec[k] for k in ("roofline", "e2e", "parity", "configs", "surrogate", "implicit_step"))


def test_line_without_the_optional_blocks():
    rec = {k: v for k, v in record().items()}
    for k in ("configs", "surrogate", "implicit_step", "e2e", "parity", "cpu_baseline"):
        rec[k] = None
    line, detail = bench.split_record(rec)
    json.dumps(line)
    assert set(detail) == {"roofline"} and line["e2e"] is None
