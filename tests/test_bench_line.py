"""bench.py's result line keeps every key a reader of it needs and stays short
however much the run records beside it."""
import json
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

import bench  # noqa: E402

REQUIRED = ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
            "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "clocks")


def test_line_is_short_and_complete():
    number = 123456.78901234567
    stages = {k: number for k in ("split_prep", "assembly", "minors", "cdet")}
    note = "x" * 400
    line = dict.fromkeys(REQUIRED, number)
    line.update(metric=bench.METRIC, dtype="f64 (split fp16-digit tcgen05 assembly, FP64 minors and CDet)",
                data="synthetic (seeded uniform vertices, tables from the in-tree precompute)",
                config=bench.line_config("split", 1), vs_baseline=None,
                e2e={"value": number, "unit": bench.UNIT, "h2d_bytes_per_step": 21233664, "d2h_bytes_per_step": 786432},
                clocks={"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": ["sw_power_cap"], "samples": 41},
                stages_ms_per_step=stages, flagged_configs=0, e2e_bit_identical=True, split_over_fp64=number,
                roofline={"kernel": "split_assembly (tcgen05 fp16 digit slices)", "bound": "tensor",
                          "achieved": number, "peak": number, "unit": "TFLOP/s", "frac": number, "traffic": number,
                          "note": note},
                fp64_path={"value": number, "ms_per_step": number, "bit_identical_to_reference": True, "stages": stages},
                dd_path={"note": note}, cpu_baseline={"value": number, "unit": "configs/s", "cores": 16, "kind": "port",
                                                      "sample": note},
                precision_by_order={"worst_condition_scaled": number, "contract_met": True,
                                    "orders": {str(n): {"note": note * 4} for n in range(1, 11)}})
    line["at_1e-10_relative"] = {"value": number, "ms_per_step": number, "worst_relative_error_orders_2_10": number,
                                 "contract_met": True, "form": note}
    out = bench.headline(line)
    assert all(k in out for k in REQUIRED)
    assert len(json.dumps(out)) < 2500
    assert all(out[k] == line[k] for k in REQUIRED)


def test_line_without_the_optional_parts():
    line = dict.fromkeys(REQUIRED, 1.0)
    assert bench.headline(line) == line
