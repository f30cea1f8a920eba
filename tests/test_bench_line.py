"""The benchmark's printed record: the keys a reader needs, and short enough to
be read back from the end of a log (every step time and check made it 30 KB)."""
import json
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)


def test_printed_record_is_short_and_keeps_the_largest_errors():
    import bench

    l1 = {k: 1.234567890123e-08 for k in ("rho", "mx", "my", "mz", "E")}
    checks = [{"step": i, "dt_gpu": 5.5e-7, "dt_oracle_rel_diff": 0.0,
               "fp64": dict(l1, rho=1e-17 * (i + 1)), "fp32_bulk": dict(l1, my=1e-8 * i)} for i in range(20)]
    sample = [{"problem": "ensemble[%d] side 16" % i, "rel_l1": l1, "steps": 50, "oracle_steps": 50,
               "t_rel_diff": 1e-16 * i} for i in range(5)]
    point = {"offered_load_of_burst": 0.25, "rate_hz": 23.8, "latency_p50_s": 0.0127648, "latency_p99_s": 0.1057,
             "cell_updates_per_s": 4063023877.617, "makespan_s": 4.37, "requests": 100}
    leg = {"value": 6284938967.588052, "ms_per_coarse_step": 0.72188704, "ms_each_step": [0.712] * 200}
    line = {"metric": "m", "value": 20949102345.678, "unit": "cell-updates/s", "n_gpus": 1, "ms_per_step": 0.8008561,
            "config": {"workload": "sedov3d_256", "cells": 16777216}, "gpu_launches": 20,
            "e2e": {"value": 928948664.0904772, "unit": "cell-updates/s", "h2d_bytes_per_step": 671088640},
            "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": []},
            "amr": {"workload": "w" * 90, "fp64": leg, "fp32_bulk": leg, "per_step_vs_oracle": checks,
                    "fp32_bulk_vs_fp64_trajectory_rel_l1": [dict(l1, after_steps=10 * i) for i in range(19)]},
            "batch": {"results_vs_oracle": {"fp32_bulk": sample, "fp64": sample}},
            "serve": {p: {"load_sweep": {"points": [point] * 4}} for p in ("fp32_bulk", "fp64")}}
    assert len(json.dumps(line)) > 15000
    out = bench.printed(line)
    assert len(json.dumps(out)) < 4000
    assert set(out) == set(line)
    for k in ("metric", "unit", "n_gpus", "config", "gpu_launches", "clocks"):
        assert out[k] == line[k]
    assert abs(out["value"] / line["value"] - 1) < 1e-5 and out["e2e"]["unit"] == "cell-updates/s"
    c = out["amr"]["per_step_vs_oracle"]
    assert c["checks"] == 20 and c["fp64_rel_l1_rho"] == 2e-16 and c["fp32_bulk_rel_l1_others"] == 1.9e-7
    assert out["batch"]["results_vs_oracle"]["fp64"]["t_rel_diff"] == 4e-16
