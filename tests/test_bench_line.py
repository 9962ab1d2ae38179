"""bench.py's printed line: short whatever was measured, with every number that its reader looks for."""
import json

import sys
from pathlib import Path

sys.path.insert(0, str(Path(__file__).resolve().parents[1]))
import bench  # noqa: E402

FORM = {"views_per_s": 2676.519, "e2e_views_per_s": 2650.1, "passes_ms": {f"pass {k}": 0.1234 for k in range(7)},
        "tune_table": [{"views_per_frame": k, "views_per_s": 1234.567} for k in range(60)],
        "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": []}}


def _line():
    return {
        "metric": bench.METRIC, "value": 2676.519, "unit": bench.UNIT, "n_gpus": 8, "steps": 20, "warmup": 5,
        "ms_per_step": 112.086, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
        "data": "synthetic",
        "config": {"workload": "learned_1080p", "gaussians": 1_240_000, "resolution": "1920x1080",
                   "scene_format": "f32/soa", "bounds": "tight", "list": "adaptive, binning (depth sort, then by tile rows)",
                   "form": "batched (16 views per frame) + learned colour (fp16 latent, BF16 MLP, 100.0% SH fallback at the "
                           "2/255 gate)", "step": "one pass over the 300-view orbit (r=14, h=2)",
                   "l2": "inputs larger than L2 (scene 298 MB), no flush", "cuda_graph": True,
                   "parallelism": "replicas x8 (orbit workloads); views split by pixel count (batched_64, scale_4k)"},
        "views_timed": 48_000,
        "e2e": {"value": 2650.123, "unit": bench.UNIT, "h2d_bytes_per_step": 32_400, "d2h_bytes_per_step": 1_866_240_000},
        "gpu_launches": 4180, "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": ["sw_power_cap"]},
        "speedup_vs_plain": 1.2881,
        "roofline": {"bound": "hbm", "kernel": "preprocess + sort " * 8, "achieved": 2513.1, "peak": 6453.1, "unit": "GB/s",
                     "frac": 0.3894, "peak_kind": "measured", "algorithmic_bytes": 4_390_000_000, "ms": 1.7468,
                     "traffic": 4_350_000_000, "kernels": {f"kernel {k}": {"bytes": 1, "ms": 0.1} for k in range(9)},
                     "plain_view": {"kernels": {f"kernel {k}": {"bytes": 1, "ms": 0.1} for k in range(9)}}},
        "render_issue": {"frac": 0.8}, "issue": {"render": {"frac": 0.8}}, "render_flops": {"frac_kernel": 0.2},
        "parity": {"list_bit_exact": True, "entries": 5_184_815, "psnr_float_db": 120.6, "psnr_8bit_db": 98.8,
                   "note": "x" * 300},
        "configs": {w: {f: FORM for f in ("plain", "batched", "gated", "forced", "forced tcgen05")} | {"parity": {"a": "b" * 500}}
                    for w in bench.WORKLOADS},
        "cpu_baseline": {"value": 0.9232, "unit": "views/s", "cores": 16, "kind": "port",
                         "sample": "10 of 300 views (every 30th), tight bounds, renderReference with 16 threads, 10.8 s"},
        "wall_s": 131.1}


def test_the_printed_line_is_short_and_whole():
    line = _line()
    out = bench.headline(line)
    text = json.dumps(out)
    assert "\n" not in text and len(text) < 3000 < len(json.dumps(line))
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling", "vs_baseline",
              "dtype", "data", "config", "e2e", "gpu_launches", "clocks", "cpu_baseline"):
        assert out[k] == line[k], k
    assert out["configs"]["plain_720p"]["batched"] == 2676.519 and "parity" not in out["configs"]["plain_720p"]
    assert out["roofline"]["frac"] == 0.3894 and out["parity"]["list_bit_exact"] is True


def test_a_single_workload_has_its_line_too():
    line = {k: v for k, v in _line().items() if k not in ("roofline", "parity", "cpu_baseline")}
    line["configs"] = {"plain_720p": {"plain": FORM, "parity": None}}
    assert bench.headline(line)["configs"] == {"plain_720p": {"plain": 2676.519}}
