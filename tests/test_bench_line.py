"""The benchmark's printed line: the contract's keys, and short enough to survive as the end of an output."""
import json
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))


def test_headline_is_short_and_whole():
    import bench
    x = 1.0 / 3.0e-12
    vs = {"oracle": x, "oracle_se": x, "error": x, "combined_se": x, "error_in_se": -x, "oracle_kind": "o" * 200}
    run = {"options_per_s": x, "time_s": x, "rounds": 58}
    book = {"batched": run, "plain": run, "checks": {"sample": [vs] * 16}, "converged": 3}
    full = {"metric": "path-steps/s", "value": x, "unit": "path-steps/s", "n_gpus": 8, "steps": 20, "warmup": 5,
            "ms_per_step": x, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
            "data": "synthetic", "config": {"workload": "w" * 130, "l2": "f" * 70, "seq_len": 256},
            "price_check": x, "price_check_se": x, "vs_oracle": vs, "geom_check": {"price": x, "vs_closed_form": vs},
            "orderings": {k: {"value": x, "ms_per_step": x, "vs_oracle": vs} for k in ("bridge", "pca_tcgen05")},
            "e2e": {"value": x, "unit": "path-steps/s", "h2d_bytes_per_step": 264, "d2h_bytes_per_step": 2560,
                    "what": "w" * 300, "ms_per_run": x, "n_samples": 1 << 23, "converged": True, "vs_oracle": None},
            "roofline": {"bound": "fp32", "achieved": x, "peak": x, "unit": "TFLOP/s", "frac": x, "traffic": 599296,
                         "note": "n" * 300},
            "gpu_launches": 40, "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": ["sw_power_cap"]},
            "book": dict({k: book for k in ("eps_1e-3_all", "eps_1e-3", "own_eps", "eps_5e-3", "mixed")}, options=256),
            "other_workloads": {"workload_number_%d" % i: {"time_s": x, "price": x, "vs_oracle": vs} for i in range(4)},
            "cpu_baseline": {"value": x, "unit": "path-steps/s", "cores": 16, "kind": "port", "sample": "s" * 80}}
    line = bench.headline(full)
    assert len(json.dumps(line)) < 2500
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
              "vs_baseline", "dtype", "data", "config", "gpu_launches", "clocks", "cpu_baseline"):
        assert line[k] == full[k]
    assert all(line["e2e"][k] == full["e2e"][k] for k in ("value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"))
    assert line["book_options_per_s"]["mixed"] == [float("%.6g" % x)] * 2
    for k in ("book", "other_workloads", "cpu_baseline"):   # each may be left out
        full.pop(k)
    assert len(json.dumps(bench.headline(full))) < 2500
