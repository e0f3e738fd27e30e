"""The line that bench.py prints: the contract's keys, and short enough that an
output's last two thousand characters hold it, whatever the blocks that go to
--details grow to."""
import json

import bench


def _full():
    big = {f"key_{k}": [k / 7.0] * 50 for k in range(200)}
    number = 10915234.123456789
    config = {k: number for k in bench.CONFIG_KEYS}
    config |= {"workload": "fe15648_1024x1024", "bounds": "workload's own",
               "sample": "4096 seeded pixels of the map (same in both arms)",
               "parallelism": "pixel shards x8",
               "l2": "inputs larger than L2 (2 GB of profiles per GPU)",
               "converged_sample": "4096 seeded pixels vs the reference FP64 chi^2",
               "histograms": big, "autotuned": big, "plain_lm": big, "initialiser_gemm": big}
    return {
        "metric": bench.METRIC, "value": number, "unit": bench.UNIT, "n_gpus": 8, "steps": 20,
        "warmup": 5, "ms_per_step": 95.61234567890123, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f32+f64 (MLP bf16)",
        "data": "synthetic (seeded draws of the workload's parameter distributions, GPU "
                "FP64 synthesis + Gaussian noise; sample pixels synthesised on the host)",
        "config": config, "plain_converged_pixels_per_s": number, "learned_vs_plain": 3.1,
        "parity_all_pass": True, "gpu_launches": 24980,
        "e2e": {"value": number, "unit": bench.UNIT, "h2d_bytes_per_step": 2013265920,
                "d2h_bytes_per_step": 83886080, "h2d_ms": 36.211647033691406,
                "d2h_ms": 17.9682559967041, "steps": 1, "warmup": 1,
                "host_buffers": "page-locked (profiles streamed in chunks)"},
        "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "samples": 260,
                   "reasons": ["hw_slowdown", "hw_thermal_slowdown", "sw_power_cap"]},
        "roofline": {k: number for k in bench.ROOFLINE_KEYS}
        | {"note": "n" * 600, "kernels": big},
        "cpu_baseline": {"value": number, "unit": bench.UNIT, "cores": 16, "kind": "reference",
                         "sample": "4096 seeded pixels of the map, 16 processes of the "
                                   "reference core"},
        "parity": big, "other_workloads": big, "stats": big}


def test_line_is_short_and_complete():
    full = _full()
    text = bench.stdout_line(full)
    assert len(text) <= bench.LINE_LIMIT and "\n" not in text
    line = json.loads(text)
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step",
                "higher_is_better", "scaling", "vs_baseline", "dtype", "data", "config", "e2e",
                "gpu_launches", "clocks", "roofline", "cpu_baseline"):
        assert key in line
    assert abs(line["value"] / full["value"] - 1) < 1e-6
    assert line["e2e"]["h2d_bytes_per_step"] == 2013265920
    assert line["config"]["workload"] == "fe15648_1024x1024"
    assert full["stats"] and full["config"]["histograms"]  # the whole is left alone
