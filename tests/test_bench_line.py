"""The benchmark prints one line that a reader of its last three thousand characters gets whole, with every key that the
workload's figure needs, whatever the other workloads' records hold."""
import json

import pytest

import bench


def record(big):
    reps = [{"ctor_ms": 12.25, "compute_ms": 2291.712345, "total_ms": 2304.9}] * 6
    acc = {f"after_{k}_steps": {"particles": 4096, "cell_rms": 1.23456789012e-5, "cell_p50": 1e-6, "cell_p99": 0.1,
                                "cell_max": 2.0} for k in (100, 400, 2000)}
    parity = {"f32_bitexact": True, "checks": {"positions": True}, "sample": 4096, "records": 201, "mismatched_particles": 0,
              "status_vs_f64_differ": 3, "f64": acc}
    e2e = {"value": 3492552040.992335, "unit": "particle-steps/s", "h2d_bytes_per_step": 5712059136,
           "d2h_bytes_per_step": 4020000000, "steps": 5, "ms_per_step": 209.87376519999825, "particle_steps": 10 ** 10,
           "reps": reps, "parity": parity, "host_buffers": "x" * 90}
    return {
        "metric": "particle-steps/s", "value": 10143042234.604431, "unit": "particle-steps/s", "n_gpus": 1, "steps": 20,
        "warmup": 5, "ms_per_step": 72.26579856872559, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "f32", "data": "synthetic (seeded Fourier-mode field)",
        "config": bench.plain_config(type("A", (), dict(sim_steps=2000, particles=10 ** 6, storage="f32", sort_interval=8,
                                                        steps_per_launch=0, layout=0)), 1),
        "run": {"records": 201, "steps_run": 2000, "particle_steps_per_run": 732993047},
        "parity": parity, "e2e": dict(e2e, pageable=e2e), "native_loader": {"value": 4.2e9 / 3, "unit": "particle-steps/s",
                                                                            "run_ms": 94.61955261230469, "path": "y" * 150},
        "roofline": {"bound": "hbm", "achieved": 9336.157404309313, "peak": 6529.1, "unit": "GB/s", "frac": 1.4299302207516063,
                     "traffic": 115446719.9025, "peak_source": "measured", "bytes_per_particle_step": 850,
                     "bytes_note": "z" * 150, "kernel": "advance_kernel<3,RK4,Pair<float>>", "avg_launch_ms": 0.3336735677048564,
                     "particle_steps_per_launch": 3664975.235, "dram_gbs": 1 / 3, "issue_frac": 2 / 3,
                     "active_bound": "issue (instruction throughput)"},
        "cpu_baseline": {"value": 23972499.91249189, "unit": "particle-steps/s", "cores": 16, "kind": "port",
                         "sample": "1000000 particles x 200 RK4 steps of the same workload (float64 oracle)"},
        "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": ["sw_power_cap"], "samples": 8}, "gpu_launches": 14000,
        "wall_s": 1.4621564669999998,
        "forms": {n: {"value": 1e10 / 3, "phase_s": 67.247770684, "accuracy": ["w" * 100] * big}
                  for n in ("gyre", "options", "precision", "batch", "serve")} if big else None,
    }


@pytest.mark.parametrize("big", [0, 1, 200])
def test_the_line_is_short_and_whole(big):
    full = record(big)
    text = json.dumps(bench.headline(full))
    assert len(text) <= bench.LINE_LIMIT and "\n" not in text
    line = json.loads(text)
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
                "vs_baseline", "dtype", "data", "config", "clocks", "gpu_launches"):
        assert line[key] == full[key], key
    assert line["e2e"]["value"] == full["e2e"]["value"]
    for key in ("unit", "h2d_bytes_per_step", "d2h_bytes_per_step"):
        assert line["e2e"][key] == full["e2e"][key]
    assert line["roofline"]["frac"] == pytest.approx(full["roofline"]["frac"], rel=1e-5)
    assert "cpu_baseline" in line
    if big:
        assert line["forms"]["serve"]["value"] == pytest.approx(1e10 / 3, rel=1e-5)


def test_the_line_stays_short_without_room():
    full = record(1)
    full["config"]["note"] = "v" * 900
    assert len(json.dumps(bench.headline(full))) <= bench.LINE_LIMIT


def test_parts_that_were_not_measured():
    full = dict(record(0), parity=None, e2e=None, native_loader=None, cpu_baseline=None)
    line = bench.headline(full)
    assert line["value"] == full["value"] and line["e2e"] is None
