"""CPU test of the line bench.py prints: one line of a few KB with the headline whole, whatever the
other sections hold; those go to the details file, complete."""
import io
import json
from contextlib import redirect_stdout

import bench


def run():
    tuning = {"chosen": "128x6", "ms_per_step": {f"{b}x{m}": 0.1 * m for b in (64, 128, 256) for m in range(12)}}
    forms = {f: {"value": 1.9e9, "ms_per_step": 0.3357181451970881, "returns": 62697973} for f in ("fp32k", "fp32k_mlp", "fp64")}
    return {
        "metric": bench.METRIC, "value": 2.44e9, "unit": bench.UNIT, "n_gpus": 1, "steps": 20, "warmup": 5,
        "ms_per_step": 1.7192, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32k",
        "data": "synthetic", "config": {"workload": "w" * 300, "particles": 4_194_304},
        "roofline": {"bound": "hbm", "achieved": 848.0}, "compute": {"pipe": "fp32"},
        "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": []}, "gpu_launches": 120,
        "stage_ms": {f"stage {k}": 0.1 * k for k in range(7)}, "status": 0, "launch_tuning": tuning,
        "e2e": {"value": 5.6e8, "unit": bench.UNIT, "h2d_bytes_per_step": 1, "d2h_bytes_per_step": 1},
        "fp64": {"value": 1.4e9, "ms_per_step": 3.04, "stage_ms": {"a": 1.0}, "roofline": {"bound": "hbm"}},
        "batched_sweep": {"ms_per_step": 2.9149, "autotune": {"table": ["x" * 100] * 50},
                          "sweep_run": {"ms_per_step": 2.92, "reference_runs": ["y" * 100] * 50}},
        "config3_run": {"ms_per_step": {"fp64": 1.98, "fp32k": 0.3357}, "curve": [[k, 0.1] for k in range(3000)]},
        "learned_warm_start": {**forms, "workload": "z" * 200},
        "ti64_cut_small": {**forms, "launch_tuning": tuning},
        "cpu_baseline": {"value": 4.6e6, "unit": bench.UNIT, "cores": 16},
    }


def test_short_line_and_whole_details(tmp_path):
    line = run()
    assert len(json.dumps(line)) > 30_000
    buf = io.StringIO()
    with redirect_stdout(buf):
        bench.emit(line, tmp_path / "details.json")
    printed = buf.getvalue()
    assert printed.count("\n") == 1 and len(printed) < 6000
    short = json.loads(printed)
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
              "vs_baseline", "dtype", "data", "config", "e2e", "clocks", "gpu_launches", "roofline", "cpu_baseline"):
        assert short[k] == line[k], k
    t = short["sections_ms_per_step"]
    assert t["fp64"] == 3.04 and t["batched_sweep"] == {"": 2.9149, "sweep_run": 2.92}
    assert t["config3_run"] == {"fp64": 1.98, "fp32k": 0.3357}
    assert t["learned_warm_start"]["fp32k_mlp"] == t["ti64_cut_small"]["fp32k_mlp"] == 0.335718
    assert json.loads((tmp_path / "details.json").read_text()) == line


def test_details_that_cannot_be_written(tmp_path, capsys):
    bench.emit(run(), tmp_path / "missing" / "details.json")
    out = capsys.readouterr()
    assert json.loads(out.out)["value"] == 2.44e9 and "not written" in out.err
