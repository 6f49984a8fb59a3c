"""bench.py's JSON line stays short: the configurations beside the headline one are carried in brief."""
import json

import bench


def test_configurations_are_brief_and_keep_their_figures():
    full = {
        "value": 123456.78901234567, "ms_per_step": 1.2345678901234567, "steps": 20, "blocks": 70, "timed_region_s": 1.1,
        "block_ms_per_step": {"min": 1.0, "median": 1.1, "max": 1.2},
        "e2e": {"value": 98765.43210987654, "unit": "QPS", "h2d_bytes_per_step": 1234567890, "d2h_bytes_per_step": 117440512,
                "ms_per_step": 1.3, "blocks": 60, "timed_region_s": 1.0, "api": "x" * 60},
        "gpu_launches": 5600,
        "roofline": {"bound": "tensor", "achieved": 2653.9426651765316, "unit": "TFLOP/s", "frac": 0.9513703273503483,
                     "peak_source": "x" * 300},
        "kernels": {"gemms": {"avg_ms": 1.0, "tops": 1.0}, "pack_gemm": {"avg_ms": 0.4}, "scan_after_pack": {"avg_ms": 0.6},
                    "tail": {"avg_ms": 0.05}, "batches_timed": 5},
        "plain_per_query": {"qps": 750.6825540898951, "queries": 32, "p50_ms": 1.33, "p99_ms": 1.34, "api": "x" * 80,
                            "batched_over_plain": 1.04},
        "byte_exact": {"device_vs_host_path": True, "plain_vs_batched": True},
        "config": {"workload": "x" * 150, "rows": 2097152, "record_bytes": 32768, "batch": 1024, "l2": "x" * 120},
        "clocks": {"sm_mhz": 1702.0, "reasons": ["sw_power_cap"], "samples": 11}, "lanes": 1, "vs_baseline": 62.9,
        "vs_baseline_ref": "x" * 60,
    }
    short = bench.brief(full)
    assert len(json.dumps(short)) < 1000
    assert short["value"] == full["value"] and short["e2e"]["value"] == full["e2e"]["value"]
    assert short["config"] == {"rows": 2097152, "record_bytes": 32768, "batch": 1024}
    assert short["roofline"]["frac"] == full["roofline"]["frac"] and short["byte_exact"] == full["byte_exact"]
