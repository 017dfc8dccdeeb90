"""The line that bench.py prints for the headline run: short enough to be read
back from a log's tail, with every key of its contract."""
import json
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

import bench  # noqa: E402

CONTRACT = ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
            "vs_baseline", "dtype", "data", "config", "e2e", "clocks", "gpu_launches")


def test_printed_line_is_short_and_complete():
    v = 101912345.678901234
    long = "the words that explain a row " * 20
    line = {"metric": bench.METRIC, "value": v, "unit": "translations/s", "n_gpus": 1, "steps": 20, "warmup": 5,
            "ms_per_step": 19.62469104766846, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "x" * 150, "data": "synthetic (seeded P2M of random charges)",
            "config": {"workload": "w" * 200, "global_batch": 2000000, "parallelism": "replica1", "l2": "l" * 60},
            "plain_fp64": {"value": v, "ms_per_step": v}, "split_over_plain_fp64": 1.1578901234,
            "split_ff": {"value": v, "ms_per_step": v, "note": long},
            "accuracy_vs_fp64_oracle_1000": {k: {"rel_l2_orthonormal_max": 3.6364e-9, "per_degree": [v] * 16}
                                             for k in ("plain_fp64", "split", "split_ff", "tc_tf32x3", "tc_bf16x3", "tc_bf16x6")},
            "physics_checks": {"what": long, "rows": [{"a": v}] * 30},
            "e2e": {"value": v, "unit": "translations/s", "h2d_bytes_per_step": 4688000000,
                    "d2h_bytes_per_step": 4352000000, "api": long},
            "e2e_classic_call": {"value": v, "api": long},
            "tensor_core": {n: {"value": v, "roofline": {"note": long}} for n in ("tc_tf32x3", "tc_bf16x3", "tc_bf16x6")},
            "roofline": {"bound": "hbm", "achieved": v, "peak": v, "unit": "GB/s", "frac": 0.1, "traffic": v,
                         "traffic_source": long, "peak_source": "measured", "kernel": "k", "frac_definition": long},
            "cpu_baseline": {"value": v, "unit": "translations/s", "cores": 16, "kind": "reference", "sample": long},
            "clocks": {"sm_mhz": 1845.0, "sm_max_mhz": 2070.0, "reasons": ["sw_power_cap"]}, "gpu_launches": 20,
            "configs": {"mixed": long}}
    out = bench.summary(line)
    assert len(json.dumps(out)) < 2000
    for k in CONTRACT:
        assert k in out, k
    assert out["value"] == v and out["ms_per_step"] == line["ms_per_step"]
    assert out["e2e"]["h2d_bytes_per_step"] == 4688000000 and out["e2e"]["d2h_bytes_per_step"] == 4352000000
    assert out["error_vs_fp64_oracle"]["split"] == 3.6364e-9
    assert out["clocks"] == line["clocks"] and out["config"] == line["config"]
