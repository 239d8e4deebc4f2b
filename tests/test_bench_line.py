"""bench.py's headline line carries its contract's keys and stays short enough
to be read whole from the last 2.9 KB of a captured output; everything else is
in a second record."""
import json
import sys
from pathlib import Path

import pytest

sys.path.insert(0, str(Path(__file__).resolve().parent.parent))


def test_headline_line_is_short_and_complete():
    pytest.importorskip("torch")
    import bench

    x = 1.2345678901234567e-06
    errs = {"max_rel": x, "frob_rel": x, "max_elem_rel": x}
    res = {
        "value": 645.5102945924065, "ms_per_step": 1.703321599960327, "headline": "bf16x3", "gpu_launches": 60,
        "e2e": {"value": 246.16, "unit": "TFLOP/s", "h2d_bytes_per_step": 805306368, "d2h_bytes_per_step": 268435456,
                "ms_per_step": 4.466521453857422, "link": {"h2d_gbs": 211.2, "note": "n" * 400}},
        "roofline": {"bound": "tensor", "achieved": 716.6071961735647, "peak": 632.6, "unit": "TFLOP/s",
                     "frac": 1.1327967059335515, "traffic": 3163000000.0, "kernel": "bf16x3_gemm",
                     "kernel_avg_ms": 1.53432959318161, "peak_source": "p" * 80,
                     "frac_of_bf16_peak_tensor_work": 1.1327967059335515},
        "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "sm_mhz_min": 2070.0, "reasons": ["sw_power_cap"],
                   "samples": 30, "window": "timed region (0.018 s), NVML every 5 ms", "power_w_max": 303.177},
        "err_vs_fp64": {"form": "bf16x3", "polybench_inputs": errs, "uniform_inputs": errs, "timed_output": errs},
        "matched_error": {"criterion": "c" * 110, "forms_meeting_it": ["tf32x3", "bf16x6", "fp16x3"],
                          "fp32_tflops": 64.50983453677901, "form": "fp16x3", "tflops": 602.4082174476741,
                          "vs_fp32": 9.338238452684651},
        "tiers": {f: {"tflops": 1.0, "more": "m" * 300} for f in bench.DTYPE_OF_FORM},
        "device": {"sm_count": 152, "cc": (10, 3)}, "peak_kind": "measured", "grouped": {"x": "g" * 2000},
        "family": {"x": "f" * 4000}, "neighbours": {"x": "n" * 4000}, "small_k": {"x": "s" * 4000},
    }
    base = {"metric": "m" * 85, "unit": "TFLOP/s", "n_gpus": 1, "steps": 20, "warmup": 5, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "data": "synthetic (analytic polybench init)",
            "config": {"workload": "w" * 110, "size": 8192, "flops_per_step": 2 * 8192 ** 3, "l2": "l" * 110,
                       "parallelism": "replicas x1"}}
    cpu = {"value": 0.137, "unit": "TFLOP/s", "cores": 16, "kind": "port", "sample": "s" * 150}
    line, details = bench.output_records(base, res, cpu)
    assert len(json.dumps(line)) < 2900
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
                "vs_baseline", "dtype", "data", "config", "clocks", "e2e", "gpu_launches"):
        assert key in line
    for key in ("value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"):
        assert key in line["e2e"]
    assert details["e2e_link"]["h2d_gbs"] == 211.2 and set(details["tiers"]) == set(bench.DTYPE_OF_FORM)
    for key in ("grouped", "family", "neighbours", "small_k", "device"):
        assert details[key] == (res[key] if key != "device" else {"sm_count": 152, "cc": [10, 3]})
