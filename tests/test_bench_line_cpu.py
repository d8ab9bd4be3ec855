"""bench.py prints one JSON line that a reader of the last 3,000 characters can
parse, with the fields it must have, however much the run recorded."""
import json
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

import bench  # noqa: E402


def _section(name):
    x = 1234567890.123456789
    return {"metric": "atom-timesteps/s", "value": x, "unit": "atom-timesteps/s", "n_gpus": 1, "steps": 1000,
            "warmup": 20, "ms_per_step": x, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "f32-pair/f64-state", "data": "synthetic (seeded FCC lattice, Maxwell-Boltzmann velocities)",
            "config": {"workload": name, "description": bench.WORKLOADS[name]["desc"], "atoms": 16_777_216,
                       "precision": "mixed", "thermo_every": 20, "rebuild_every": "on displacement > skin/2",
                       "neighbours_per_atom": x, "cells": [187, 187, 187], "lanes_per_atom": 16,
                       "list_entries_per_load": 4, "block": 256, "parallelism": "single-gpu",
                       "l2": "inputs larger than L2 (neighbour list 17.34 GB)", "cuda_graph": True},
            "gpu_launches": 123456, "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "samples": 999, "window": "w" * 99,
                                               "reasons": ["hw_slowdown", "sw_power_cap"]},
            "autotune_density_plus_pair_ms": {"%dx4x%d" % (a, b): [x, x] for a in (1, 2, 4) for b in range(30)},
            "roofline": {"kernel": "k_eam_rho_bonds + k_eam_force_bonds", "bound": "hbm", "achieved": x, "peak": x,
                         "unit": "GB/s", "frac": x, "binding": {"source": "s" * 300}, "kernel_ms": {"pair": x}},
            "accuracy": {"force_rel_rms_error_mixed_vs_oracle": x, "force_rel_rms_error_fp64_vs_oracle": x,
                         "oracle_atoms": "o" * 100},
            "fp64": {"value": x, "mixed_over_fp64": x, "steps": 40},
            "nve_drift": {"mixed": {"rows": [x] * 200}}, "two_level_list": {"rows": [x] * 200},
            "cpu_baseline": {"value": x, "unit": "atom-timesteps/s", "cores": 16, "kind": "port", "sample": "s" * 200},
            "e2e": {"value": x, "unit": "atom-timesteps/s", "h2d_bytes_per_step": 1207959552,
                    "d2h_bytes_per_step": 1207959552, "ms_per_step": x, "pipeline_timeline": {"marks": [[x, "in", 1]] * 200},
                    "path": "p" * 400}}


def test_line_is_short_and_complete():
    full = _section("eam_cu_4m")
    full["lj_mixture"], full["lj_fcc_32k"] = _section("lj_binary_16m"), _section("lj_fcc_32k")
    full["batched_replicas"] = {"replicas": 4096, "ms_forward_adjoint_persistent_graph": 4.3, "autotune_ms": {"a": 1.0}}
    full["parameter_adjoint"] = {"configurations": 256, "ms_per_loss_and_gradient": 0.2, "grad": {"re": 1.0}}
    text = json.dumps(bench.brief(full))
    assert "\n" not in text and len(text) < 2900 < len(json.dumps(full))
    line = json.loads(text)
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
              "vs_baseline", "dtype", "data", "gpu_launches"):
        assert k in line
    assert abs(line["value"] / full["value"] - 1) < 1e-5 and line["config"]["workload"] == "eam_cu_4m"
    assert set(line["clocks"]) == {"sm_mhz", "sm_max_mhz", "reasons"}
    assert {"value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"} <= set(line["e2e"])
    assert line["lj_mixture"]["value"] and line["lj_fcc_32k"]["ms_per_step"]


def test_line_without_optional_sections():
    full = {k: v for k, v in _section("lj_fcc_32k").items()
            if k not in ("accuracy", "fp64", "e2e", "cpu_baseline", "nve_drift", "two_level_list")}
    line = json.loads(json.dumps(bench.brief(full)))
    assert line["config"]["workload"] == "lj_fcc_32k" and "e2e" not in line
