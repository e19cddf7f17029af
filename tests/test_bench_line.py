"""The benchmark's result line, built from made-up records (CPU): the agreed keys, a row for every workload, and
short enough that the tail of a log holds all of it."""
import argparse
import json

import bench
import bench_workloads as BW


def test_result_line_is_short_and_complete():
    entry = {"calls": 20, "avg_ms": 0.126364803314209, "algorithmic_bytes": 704643072, "achieved_gbs": 5576.260584586111,
             "frac": 0.8639605510413384}
    record = {
        "workload": "x" * 90, "value": 617567501946.8988, "ms_per_step": 0.1290414015452067, "graph": True,
        "replays_per_step": 24, "timed_region_ms": 61.93987274169922, "step_frac": 0.8460401374773324, "launches_per_step": 3,
        "roofline": dict(entry, bound="hbm", kernel="k" * 40, kernels={"a" * 40: entry, "b" * 40: entry}),
        "e2e": {"value": 1.2e10, "unit": "logit elements/s", "h2d_bytes_per_step": 352321536, "d2h_bytes_per_step": 4,
                "ms_per_step": 23.5, "steps": 10},
        "l2": "x" * 90, "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": ["sw_power_cap"], "window": "x" * 80},
        "scaling": "strong", "cpu_baseline": {"value": 1.0, "sample": "x" * 80}, "reference_v3": {"ms_per_step": 11.6},
    }
    results = {name: record for name in BW.WORKLOADS}
    results["lsr"] = {"workload": "x", "error": "RuntimeError()"}
    wl = BW.WORKLOADS[BW.HEADLINE]
    line = bench.result_line(results, BW.HEADLINE, wl, wl, argparse.Namespace(steps=20, warmup=5), 1, None)
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
                "vs_baseline", "dtype", "data", "config", "roofline", "e2e", "gpu_launches", "clocks", "table"):
        assert key in line
    assert set(line["table"]) == set(BW.WORKLOADS) and line["table"]["lsr"] == "error"
    assert all(len(row) == len(line["table_columns"]) for row in line["table"].values() if row != "error")
    assert line["gpu_launches"] == 3 * 20 * 24
    assert len(json.dumps(line)) < 6000
