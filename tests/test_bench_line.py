"""bench.py's result line: everything the headline's reader needs, short enough
to be taken in whole whatever the other workloads report."""
import json
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402


def test_result_line_is_short_and_complete():
    kernels = {"kernel_%d" % k: {"launches_per_step": 3.75, "ms_per_step": 1.0 / (k + 1), "share": 0.5} for k in range(20)}
    policy = {"ms_per_batch_median": 126.27862548828125, "mats_per_s": 79191.57791961999, "gflops_credited": 2140.212858,
              "fallback_rate_of_all": 0.0, "route_fractions": [0.0, 1.0, 0.0], "policy": "x" * 300,
              "accuracy_last_batch": {"residual_rel_%d" % k: 1.085683709857537 for k in range(10)},
              "kernels_traced_one_batch": kernels}
    batch = {"count": 10000, "workload": "x" * 200, "plain_fp64": policy, "always_shifted_cholqr3": policy,
             "always_cholqr2": policy, "cholqr2_trial": policy, "learned": policy, "best_mixed_over_plain": 2.76323}
    square = {"workload": "x" * 150, "value": 15527.702885160752, "ms_per_step": 755.3, "kernels": kernels,
              "accuracy": {"res": 1e-15, "tol": 1e-10, "r_diag_abs_first_last": [1.0, 2.0]}}
    out = {"metric": bench.METRIC, "value": 5571.159575951798, "unit": "GFLOP/s", "n_gpus": 1, "steps": 16, "warmup": 4,
           "ms_per_step": 12.334797859191895, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
           "dtype": "f64", "data": "synthetic: " + "x" * 180, "config": {"workload": "x" * 300, "parallelism": "single-gpu"},
           "plain_fp64": square, "tsqr_fp64": square, "roofline": {"bound": "hbm", "frac": 0.34, "traffic_source": "x" * 150},
           "kernels": kernels, "e2e": {"value": 2125.97, "unit": "GFLOP/s", "h2d_bytes_per_step": 1,
                                       "d2h_bytes_per_step": 2, "pipeline": "x" * 500},
           "out_of_core": square, "gpu_launches": 1024, "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": []},
           "cpu_baseline": {"value": 22.5, "unit": "GFLOP/s", "cores": 16, "kind": "port", "sample": "x" * 250,
                            "cholqr_hr_leaf": square},
           "workloads": {"recursive": square, "square": {"plain": square, "mixed": square}, "batched": batch,
                         "learned": batch, "broken": {"error": "RuntimeError: x"}},
           "per_kappa_ms": {"100": 9.74, "1e+14": 16.66}, "accuracy": {"tol": 3.55e-13, "mixed": {"100": {"res": 6e-16}}}}
    line = bench.result_line(out)
    assert len(json.dumps(line)) < 6000 and "\n" not in json.dumps(line)
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
                "vs_baseline", "dtype", "data", "config", "clocks", "gpu_launches"):
        assert line[key] == out[key]
    assert {k: line["e2e"][k] for k in ("value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step")} == {
        "value": 2125.97, "unit": "GFLOP/s", "h2d_bytes_per_step": 1, "d2h_bytes_per_step": 2}
    assert line["workloads"]["square"]["mixed"] == {"value": 15528.0, "ms_per_step": 755.3,
                                                    "accuracy": {"res": 1e-15, "tol": 1e-10}}
    assert line["workloads"]["broken"] == {"error": "RuntimeError: x"}
    assert line["workloads"]["batched"]["learned"]["mats_per_s"] == 79192.0
    assert list(line)[-2:] == ["per_kappa_ms", "accuracy"]
    assert "kernels" in out  # the caller's dict is left whole
