"""The benchmark's line stays short enough to be read whole from a captured
standard output: its long explanations are split off."""
import json

import bench


def _full_line():
    e2e = {"value": 1.0 / 3, "unit": "voxel-updates/s", "h2d_bytes_per_step": 1, "d2h_bytes_per_step": 2,
           "breakdown_ms": {"device_step": 1.0 / 7, "note": "n" * 600}}
    return {
        "metric": "voxel-updates/s", "value": 1234567890123.456, "unit": "voxel-updates/s", "n_gpus": 1, "steps": 20,
        "warmup": 5, "ms_per_step": 100.0 / 3, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "f32", "data": "synthetic", "config": {"workload": "w" * 250, "path": "p" * 250},
        "fp16_storage": {"value": 1.0 / 3, "roofline": {"frac": 1.0 / 3, "note": "n" * 300}, "hu": {"x": [1.0 / 3] * 30}},
        "roofline": {"frac": 1.0 / 3}, "stages": {"rebin": {"ms_per_step": 1.0 / 3}},
        "cpu_baseline": {"value": 1.0, "sample": "s" * 500},
        "e2e": e2e, "beside": {"value": 1.0, "e2e": dict(e2e)},
        "batch": {"scans": ["d" * 70] * 24, "autotune": ["t" * 400] * 24, "batched": {"fp32": {"vs_plain": 0.98}}},
        "serve": {"scans": ["d" * 70] * 9, "per_scan_alone_ms": [1.0 / 3] * 9, "workers": 3}, "e2e_file": None,
        "gpu_launches": 132.0, "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "samples": 17, "reasons": []},
    }


def test_line_is_short_and_keeps_the_contract():
    full = _full_line()
    line, detail = bench.split_line(full)
    assert len(json.dumps(full)) > 15000 and len(json.dumps(line)) < 4000
    for k, v in full.items():
        assert k in line
        if not isinstance(v, dict):
            assert line[k] == v
    for k in ("value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"):
        assert abs(line["e2e"][k] - full["e2e"][k]) <= 1e-6 if k != "unit" else line["e2e"][k] == full["e2e"][k]
    assert set(detail) == {".".join(p) for p in bench.DETAIL}
    assert "autotune" in full["batch"], "the caller's line is not changed"


def test_lines_without_the_optional_parts():
    line, detail = bench.split_line({"metric": "m", "value": 1.5, "batch": None, "serve": None, "e2e": {"value": 2.0}})
    assert line == {"metric": "m", "value": 1.5, "batch": None, "serve": None, "e2e": {"value": 2.0}} and detail == {}
