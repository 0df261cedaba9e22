"""The benchmark's printed line stays short enough to be captured whole, and keeps what the headline is judged by."""
import json
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
import bench  # noqa: E402

NUMBER = 1234567890.1234567


def _entry():
    return {"value": NUMBER, "ms_per_step": 0.12345678901234567, "particles": 16777216, "mode": "parity",
            "precision": "mixed", "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": [], "samples": 1},
            "gpu_launches": 1234, "bed": {"kinetic_energy": NUMBER, "coordination_number": NUMBER,
                                          "solid_fraction_box": NUMBER}, "verlet_skin_m": 0.0003,
            "e2e": {"value": NUMBER, "wall_ms": NUMBER, "h2d_bytes_per_step": NUMBER, "d2h_bytes_per_step": NUMBER},
            "roofline_frac": 0.1, "force_ms": 0.2, "jkr": {"counters": dict.fromkeys("abcdefgh", 123456789)},
            "autotune": {"tried": 99, "note": "x" * 300},
            "force_err": {"force_rel_sum": 1.23456789e-10, "force_rel_net": 1e-7, "torque_rel_sum": 1e-9,
                          "method": "y" * 300}}


def _record():
    forms = {"hopper-1M": {k: _entry() for k in ("plain", "mixed", "physical")},
             "adhesive-4M": {**{k: _entry() for k in ("certified", "learned", "learned_mixed", "newton_mixed", "newton")},
                             "training": {"train_ms": 230.0}, "note": "every solver from the same settled state"},
             "drum-16M": {k: _entry() for k in ("fp64", "mixed")},
             "batched-512": {"device_loop": _entry(), "one_at_a_time": {"value": NUMBER, "boxes_timed": 16}},
             "skipped": ["adhesive newton: time budget of the run used up"]}
    return {"metric": bench.METRIC, "value": NUMBER, "unit": bench.UNIT, "n_gpus": 1, "steps": 20, "warmup": 5,
            "ms_per_step": 0.36, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic", "config": {"workload": "hopper-1M", "describe": "z" * 300, "particles": 1048576,
                                            "mode": "parity", "parallelism": "replicas x1", "l2": "inputs larger than L2"},
            "roofline": {"bound": "hbm", "achieved": NUMBER, "peak": 6787.2, "unit": "GB/s", "frac": 0.12,
                         "traffic": NUMBER, "kernel": "k" * 150, "avg_launch_ms": 0.2, "peak_source": "measured",
                         "fp64": {"achieved": NUMBER, "peak_fma_per_s": NUMBER, "frac": 0.5, "counts_source": "c" * 400}},
            "cpu_baseline": {"value": NUMBER, "unit": bench.UNIT, "cores": 16, "kind": "port", "sample": "s" * 400},
            "cpu_baseline_literal": {"value": NUMBER, "unit": bench.UNIT, "cores": 16, "kind": "port", "sample": "s" * 400},
            "e2e": {"value": NUMBER, "unit": bench.UNIT, "h2d_bytes_per_step": NUMBER, "d2h_bytes_per_step": NUMBER,
                    "note": "n" * 200, "wall_ms": NUMBER},
            "gpu_launches": 122, "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": [], "samples": 5},
            "force_err": _entry()["force_err"], "precision": "fp64", "wall_s_timed": 0.1, "stats": {"a": 1},
            "verlet_skin_m": 0.0008, "bed": {"kinetic_energy": NUMBER}, "forms": forms, "bench_wall_s": 190.1}


def test_line_is_short_and_whole():
    full = _record()
    line = bench.short_line(full)
    text = json.dumps(line)
    assert len(text) < 3500, len(text)
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
              "vs_baseline", "dtype", "data", "gpu_launches", "clocks"):
        assert line[k] == full[k], k
    assert {k: line["e2e"][k] for k in ("value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step")} == \
        {k: full["e2e"][k] for k in ("value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step")}
    assert line["config"]["workload"] == "hopper-1M" and line["config"]["particles"] == 1048576
    rows = line["forms"]["rows"]
    assert rows["drum-16M/mixed"] == [1.235e9, 0.1235, 1.235e9, 1.235e-10]
    assert rows["batched-512/one_at_a_time"][0] == 1.235e9 and rows["skipped"] == full["forms"]["skipped"]
    assert sum(isinstance(r, list) and len(r) == len(bench.FORM_COLUMNS) for r in rows.values()) == 12


def test_line_without_forms():
    full = _record()
    for k in ("forms", "cpu_baseline", "force_err"):
        full[k] = None
    full["roofline"]["fp64"] = None
    line = bench.short_line(full)
    assert "forms" not in line and line["cpu_baseline"] is None and "fp64" not in line["roofline"]
    assert json.loads(json.dumps(line))["value"] == NUMBER


def test_clock_sampler_waits_for_samples(tmp_path, monkeypatch):
    # a stand-in for nvidia-smi that starts slowly: a region shorter than its start still has samples
    fake = tmp_path / "nvidia-smi"
    fake.write_text("#!/bin/sh\nsleep 0.2\nwhile true; do echo '0, 1950, 2070, 700, 0x0, Not Active, Not Active, Not Active, Active'; "
                    "sleep 0.05; done\n")
    fake.chmod(0o755)
    monkeypatch.setenv("PATH", f"{tmp_path}:{os.environ['PATH']}")
    ck = bench.ClockSampler()
    ck.start()
    ck.wait(1)
    ck.wait(len(ck.lines) + 1, 2.0)
    got = ck.stop()
    assert got["samples"] >= 2 and got["sm_mhz"] == 1950.0 and got["sm_max_mhz"] == 2070.0
    assert got["reasons"] == ["sw_power_cap"]
