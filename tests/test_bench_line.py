"""The line that bench.py prints: short, and with every key of its contract."""

from __future__ import annotations

import json


def test_headline_is_short_and_complete():
    import bench

    rate = {"requests": 20000, "wall_s": 0.1, "offered_bytes": 10**10, "p50_ms": 12.345678901,
            "p99_ms": 99.87654321, "mean_ms": 1.0, "max_ms": 2.0, "batches": 9, "mode": "zero_copy",
            "offered_GBps": 1.23456789012345, "rate_per_s": "all at t=0", "slo_met": True}
    long = {"value": 123.4567890123456, "ms": 1.0, "note": "x" * 400}
    line = {"metric": bench.METRIC, "value": 560.1234567890123, "unit": "GB/s", "n_gpus": 1,
            "steps": 20, "warmup": 5, "ms_per_step": 0.4678901234567, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "u8", "data": "synthetic " * 6,
            "config": {"workload": bench.workload_config("c3-sustained"), "offered_bytes": 10**9,
                       "examined_bytes": 10**9, "l2": "inputs larger than L2 (no flush)",
                       "parallelism": "replicas x1", "technique": "t" * 160},
            "phases_ms": {k: 0.123456789 for k in "abcdefgh"}, "step_stats": long,
            "e2e": {**long, "unit": "GB/s", "h2d_bytes_per_step": 10**9,
                    "d2h_bytes_per_step": 24576, "ms_per_step": 1.6, "path": "p" * 300},
            "e2e_other_ingest": {"copy": long, "zero_copy": long}, "gpu_launches": 60,
            "oracle_gate": {"checked": 2048, "paths": ["copy"], "accepted": 0},
            "roofline": {**long, "bound": "smem", "achieved": 1.5, "peak": 2.5, "unit": "GB/s",
                         "frac": 0.5, "kernel": "lanes_shared_kernel", "kernel_ms": 0.38,
                         "onchip_peaks": {str(k): 1.23456789 for k in range(40)}},
            "cpu_baseline": {"value": 0.75, "unit": "GB/s", "cores": 16, "kind": "port",
                             "sample": "s" * 120},
            "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": []},
            "c1_plain_nfa": {str(k): long for k in range(10)}, "dfa_chunks": {"a": long},
            "speedup_vs_plain_per_input": 5000.123456789, "speedup_vs_plain_single_launch": 30.1,
            "serving": {"rates": [rate] * 5, "plain_per_request": long,
                        "examined_traces": {"live": {"trace": "t" * 200, "rates": [rate] * 3},
                                            "sustained": {"rates": [rate] * 5}}}}
    out = bench.headline(line)
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step",
                "higher_is_better", "scaling", "vs_baseline", "dtype", "data", "config",
                "gpu_launches", "clocks", "roofline", "cpu_baseline"):
        assert key in out
    assert out["e2e"]["value"] == long["value"] and out["e2e"]["h2d_bytes_per_step"] == 10**9
    assert [r["p99_ms"] for r in out["serving"]["live"]] == [99.877] * 3
    assert len(json.dumps(out)) < 4000 < len(json.dumps(line))
    # without the optional sections too
    short = {k: v for k, v in line.items() if k not in ("serving", "cpu_baseline")}
    assert "serving" not in bench.headline(short)
