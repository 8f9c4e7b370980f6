"""The bench's line on stdout: short enough to be read back whole, with every key
that its readers look for."""
import json

import bench


def record():
    text = "128x256:sediment*14;256x512:sediment*14;384x768:sediment*12;512x1024:sediment*24"
    leg = {f"key_{k}": 1.0 / (k + 3) for k in range(40)}
    return {
        "metric": bench.METRIC, "value": 25853123456.789123, "unit": bench.UNIT, "n_gpus": 1,
        "steps": 20, "warmup": 5, "ms_per_step": 0.7123039960861206, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": {"workload": "ensemble64", "cases": 64, "cells_per_step": 18415616,
                   "precision": "f32", "l2": "working set > L2 (129 MB)",
                   "parallelism": "case-parallel replicas x1", "plan_groups": 2},
        "roofline": {"bound": "hbm", "achieved": 2871.365937957729, "peak": 6791.4,
                     "unit": "GB/s", "peak_source": "measured hbm", "kernel": "z_transforms",
                     "frac": 0.4227944, "kernel_ms": 0.23, "traffic": None,
                     "traffic_unit": "bytes per step of the kernel's launches (ncu dram)"},
        "phase_ms": leg, "kernel_ms": leg, "plain_fp64": {"dct": leg, "dense": leg},
        "tuning": {"key": text, "trials_ms": leg},
        "e2e": {"value": 22728369585.608913, "unit": bench.UNIT, "h2d_bytes_per_step": 73662464,
                "d2h_bytes_per_step": 73674752, "groups": 2, "pipelined": "per-group graphs"},
        "gpu_launches": 320, "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": []},
        "status_ok": True, "serving": {"config": leg, "summary": leg, "steps": 9574},
        "cpu_baseline": {"value": 58729704.879678346, "unit": bench.UNIT, "cores": 16,
                         "kind": "port", "sample": text * 6, "one_core": leg},
    }


def test_line_is_whole_within_the_last_3000_characters(capsys):
    full = record()
    assert len(json.dumps(full)) > 5000
    bench.emit(full)
    out, err = capsys.readouterr()
    assert len(out) <= 2500 and out.count("\n") == 1
    line = json.loads(out)
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step",
              "higher_is_better", "scaling", "vs_baseline", "dtype", "data", "config", "e2e",
              "gpu_launches", "clocks"):
        assert k in line
        if isinstance(full[k], float):
            assert abs(line[k] - full[k]) <= 1e-6 * abs(full[k])
    assert line["config"] == full["config"]
    assert line["e2e"]["h2d_bytes_per_step"] == 73662464
    assert line["cpu_baseline"]["cores"] == 16
    assert set(line) | set(line["omitted"]) >= set(full)
    assert json.loads(err) == full


def test_short_lines_stay_whole():
    line = {k: v for k, v in record().items() if k in bench.LINE_KEYS}
    assert set(bench.compact(line)) == set(line)
