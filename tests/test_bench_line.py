"""The bench's printed line stays short enough for a log's tail, whatever number
of steps its error record covers, and holds the contract's keys."""
import json
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)


def record(steps):
    stages = {k: 0.123456789 for k in ("distributor", "poisson", "pcg", "efield", "push_move_update_deposit", "injector",
                                       "sort")}
    long_run = {"steps": 500, "first_step": 161, "value": 4181967714.7, "unit": "particle-steps/s",
                "ms_per_step": 4.7637, "particles_first": 19945760, "particles_last": 19912162,
                "pcg_iterations_per_step": 17.0, "timing": "t" * 90}
    tuning = {"threads": 512, "blocks_per_sm": 16, "dep_agg": 0, "sort_interval": 20, "pass_ms": 1.9068639874458313,
              "sort_ms": 2.1939520835876465, "amg_theta": 0.01, "amg_pcg_ms": 3.314458648363749}
    particles = {"value": 15793948147.1, "unit": "particle-steps/s", "ms_per_step": 1.2621, "stages": list(stages)[:3]}
    roof = {"bound": "hbm", "kernel": "k" * 80, "achieved": 2820.5, "peak": 6787.2, "unit": "GB/s", "frac": 0.4156,
            "peak_source": "p" * 40, "traffic": 10463000000, "algorithmic_bytes": "a" * 200, "traffic_source": "s" * 110,
            "traffic_unit": "u" * 60}
    cpu = {"value": 3711704.3, "unit": "particle-steps/s", "particle_stages_value": 5560136.1, "stage_s_per_step": stages,
           "cores": 16, "steps": 3, "amg_pcg_iterations_per_step": 37.0, "how": "h" * 150}
    errors = [1.23456789e-5 * (k + 1) for k in range(steps)]
    return {
        "metric": "m" * 90, "value": 4172464358.4, "unit": "particle-steps/s", "n_gpus": 1, "steps": 20, "warmup": 5,
        "ms_per_step": 4.777, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32+i64",
        "precision_form": "mixed", "data": "d" * 90,
        "config": {"workload": "w" * 190, "precision": "mixed", "pcg_precond": "amg", "warm_start": "prev",
                   "efield": "dg0", "step_mode": "graph", "tuning": tuning, "cells": 10362480, "dofs": 1770950,
                   "nnz": 11788382, "amg_levels": [[1770950, 11788382]] * 5, "amg_theta": 0.01,
                   "particles_initial": 19999820, "particles_mean_pushed": 19933378, "pcg_iterations_per_step": 17.0,
                   "first_timed_step": 111, "last_timed_step": 130, "l2": "l" * 90},
        "particle_stages": particles, "stage_ms_per_step": stages, "stage_share": stages, "stage_source": "s" * 50,
        "roofline": roof, "roofline_particles": roof, "roofline_pcg": roof,
        "e2e": {"value": 4088072309.5, "unit": "particle-steps/s", "h2d_bytes_per_step": 224,
                "d2h_bytes_per_step": 14167832, "path": "p" * 260, "host_buffer": "pinned"},
        "gpu_launches": 336,
        "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": ["sw_power_cap"], "samples": 80,
                   "samples_near_timed_steps": 2, "window": "w" * 80},
        "wall_s_timed": 0.096, "long_run": long_run,
        "fp64_form": {"value": 3209066175.7, "unit": "particle-steps/s", "ms_per_step": 6.203, "e2e": 3166489584.0,
                      "pcg_iterations_per_step": 17.0, "roofline_particles_frac": 0.3381, "particle_stages": particles,
                      "long_run": long_run, "stage_ms_per_step": stages, "tuning": tuning, "amg_theta": 0.01,
                      "poisson_form": "p" * 190},
        "mixed_vs_fp64": 1.3, "mixed_vs_fp64_particle_stages": 1.763,
        "rho_rel_err": {"steps": steps, "bar": 1e-5, "step0": {"l2": 4.5e-6, "max": 4.2e-6, "what": "w" * 110},
                        "interior": {"first_step_above_bar_l2": 4, "first_step_above_bar_max": 2,
                                     "l2_at_steps": {str(k): 4.33816985932561e-06 for k in (0, 9, 49, 99, 199, 499)},
                                     "what": "w" * 80},
                        "all_dofs": {"l2_median": 0.008252076241499897, "l2_max": 0.04, "max_max": 0.57},
                        "event_steps": 499, "phi_max_err": 0.0004518683184562, "per_step_l2": errors,
                        "per_step_interior_l2": errors, "per_step_max": errors,
                        "collected_current_per_species": {f: {"electrons": -0.8469163233415088, "ions": 0.26091931139}
                                                          for f in ("fp64", "mixed")},
                        "collected_current_equal_steps": 371,
                        "collected_current_rel_diff": {"electrons": 0.0001510574018128627, "ions": 0.0}, "how": "h" * 220},
        "cpu_baseline": {"value": 3711704.3, "unit": "particle-steps/s", "cores": 16, "kind": "port", "sample": "s" * 210,
                         "all_cores": cpu, "single_thread": cpu},
    }


def test_the_line_is_short_and_keeps_the_contract():
    import bench
    text = bench.line(record(500))
    assert len(text) < 5000 and "\n" not in text
    assert text == bench.line(record(500)) and len(bench.line(record(5000))) < 5000
    d, full = json.loads(text), record(500)
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
                "vs_baseline", "dtype", "data", "gpu_launches", "mixed_vs_fp64"):
        assert d[key] == full[key]
    for key in ("value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"):
        assert d["e2e"][key] == full["e2e"][key]
    for key in ("sm_mhz", "sm_max_mhz", "reasons"):
        assert d["clocks"][key] == full["clocks"][key]
    assert d["config"]["workload"] == full["config"]["workload"]
    assert d["rho_rel_err"]["step0"]["l2"] == full["rho_rel_err"]["step0"]["l2"]
    assert d["cpu_baseline"]["value"] == full["cpu_baseline"]["value"]
