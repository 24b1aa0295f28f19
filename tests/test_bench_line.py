"""The bench's JSON line, on the CPU: one line short enough to be read back from the end of a
program's output, with the run's keys unchanged; everything else in the details file."""
import json
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402

KERNELS = ("albedo", "compact_hits", "proposal_infer", "ris_candidates", "shadow_candidates", "temporal", "spatial",
           "shade_request", "shadow_shading", "shade_finish", "accumulate", "proposal_train")


def _line(method):
    """A run's line as main() builds it, with texts and numbers of their real lengths."""
    x = 2.8302863999996930
    kernels = {k: x for k in KERNELS}
    return {
        "metric": bench.METRIC, "value": x, "unit": "ms/frame", "n_gpus": 1, "steps": 250, "warmup": 5, "ms_per_step": x,
        "higher_is_better": False, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
        "data": "synthetic (seeded procedural scene)",
        "config": {"workload": "config3: " + "w" * 205, "resolution": [1920, 1080], "scene_config": 3, "l2": "l" * 130,
                   "method": method},
        "plain_ms_per_frame": x, "stage_ms": kernels, "kernel_ms": kernels, "stage_roofline": {k: kernels for k in KERNELS},
        "rays_per_frame": 5000000, "rays_per_s": 1380631281.1083908,
        "roofline": {"kernel": "shadow_candidates", "bound": "hbm", "achieved": x, "peak": 6706.5, "unit": "GB/s",
                     "frac": x, "peak_kind": "of measured", "traffic": 83360000.0, "bytes_per_launch": 68000000.0,
                     "note": "n" * 90},
        "cpu_baseline": {"value": 799.5825760000002, "unit": "ms/frame", "cores": 16, "kind": "port", "sample": "s" * 108,
                         "cpu_model": "Neoverse-V2"},
        "quality": {"points": [kernels] * 20, "learned_at_equal_mse": None},
        "e2e": {"value": x, "unit": "ms/frame", "h2d_bytes_per_step": 704, "d2h_bytes_per_step": 33177600,
                "image_ok": True, "pipelined": True, "synchronous": x, "plain_32": x, "plain_32_synchronous": x},
        "gpu_launches": 2750, "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": [], "samples": 5},
        "tuning": kernels, "tuning_search": {"tuning": kernels}, "modes": kernels, "configs_0_1": [kernels] * 4}


@pytest.mark.parametrize("method", ["m" * 42, "m" * 230])
def test_one_short_line(capsys, monkeypatch, tmp_path, method):
    monkeypatch.setattr(bench, "OUT_DIR", str(tmp_path / "out"))
    full = _line(method)
    bench.emit(full)
    printed = capsys.readouterr().out
    assert printed.count("\n") == 1 and len(printed) <= 2001
    line = json.loads(printed)
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
              "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "clocks"):
        assert line[k] == full[k], k
    assert line["plain_ms_per_frame"] == full["plain_ms_per_frame"] and line["cpu_baseline"] == full["cpu_baseline"]
    assert json.loads((tmp_path / "out" / "bench_details.json").read_text()) == full
