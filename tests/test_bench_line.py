"""bench.py's line on stdout: short enough for a reader that keeps only the end
of an output, with the keys its readers need."""
import json
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

NEEDED = ["metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
          "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "clocks", "bit_exact"]


def _full():
    x = 1234567.890123456
    served = {k: x for k in ("p50_ms", "p99_ms", "p999_ms", "max_ms", "qps", "ingest_pos_updates_per_s", "mean_batch")}
    served["server"] = {"loop": "l" * 200}
    return {
        "metric": "pos-updates/s at 10M objs (bit-exact meetings); query p50/p99 under ingest", "value": x, "unit": "u",
        "n_gpus": 1, "steps": 20, "warmup": 5, "ms_per_step": x, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f64", "data": "synthetic (seeded grid-graph traces)",
        "config": {"workload": "uniform-10M", "objects": 10_000_000, "street_grid": "200x200 over 40 km, jitter 20 m",
                   "hotspots": 0, "reach_m": 10.0, "min_meet_steps": 5, "leaf_capacity": 200,
                   "meeting_buckets": 1 << 28, "memtable": "on, flush past 134217728 directed keys, 100 CTFs, "
                   "256x256 map bitmaps", "l2": "inputs and table larger than L2; no flush", "parallelism": "replicas x1",
                   "launch_shape": {"refine_blocks_per_sm": 0}},
        "e2e": {"value": x, "unit": "pos-updates/s", "h2d_bytes_per_step": 160000000, "d2h_bytes_per_step": 38842200,
                "host_link": {"h2d_gbs": x, "d2h_gbs": x}, "windows": {"window_device_ms": [x] * 20}},
        "gpu_launches": 460, "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": [], "samples": 8},
        "roofline": {"bound": "hbm", "kernel": "sweep", "achieved": x, "peak": x, "unit": "GB/s", "frac": x,
                     "traffic_source": "t" * 100},
        "phase_ms": {n: x for n in ("partition", "border", "refine", "insert", "sweep", "schema", "copy_in", "memtable")},
        "flush": {"keys": 89943630, "ms": x, "stages_ms": {"a": x}}, "compaction": {"keys": 193886704, "ms": x},
        "sort": {"pairs": 10 ** 8, "ms": x}, "autotune": {"grid_capacity": 64, "base_step_ms": x, "best_step_ms": x},
        "batched": {"windows": 64, "failed_windows": 0, "plain_pos_per_s": x, "window_pos_per_s": x,
                    "each": [{"objects": 1, "meetings": 2}] * 64},
        "queries_under_ingest": served, "queries_under_ingest_hbm_input": dict(served), "bit_exact": True,
        "cpu_baseline": {"value": x, "unit": "pos-updates/s", "cores": 16, "kind": "port", "sample": "s" * 150},
    }


def test_the_line_is_short_and_complete():
    import bench
    line = bench.short_line(_full())
    text = json.dumps(line)
    assert len(text) < 1450 and "\n" not in text
    assert all(k in line for k in NEEDED)
    assert line["value"] == 1234567.890123456 and line["e2e"]["value"] == line["value"]
    assert line["e2e"]["h2d_bytes_per_step"] == 160000000 and line["clocks"]["reasons"] == []
    assert line["queries_under_ingest"]["p99_ms"] > 0


def test_parts_that_were_not_run_stay_null():
    import bench
    full = _full()
    for k in ("flush", "compaction", "autotune", "batched", "queries_under_ingest", "queries_under_ingest_hbm_input",
              "cpu_baseline", "bit_exact"):
        full[k] = None
    line = bench.short_line(full)
    assert line["queries_under_ingest"] is None and line["bit_exact"] is None
    assert all(k in line for k in NEEDED)
