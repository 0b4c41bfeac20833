"""The benchmark's result line is one that fits a log's tail: the per-step lists of both arms
go to the file of --detail, the line keeps what the contract and the comparison of the
arms need."""
import json

import bench


def _arm(steps):
    phases = {"davidson": 693.123456789012, "svd": 218.123456789012, "env": 65.123456789012, "gaps": 0.019123456789}
    return {"value": 10.71012345678901, "unit": "s/sweep", "ms_per_step": 450.9512345678, "s_per_update": 0.0563,
            "step_seconds": [0.45 + 1e-9 * k for k in range(steps)], "heff_tflops": 120.123456789,
            "heff_share_of_step": 0.612345678912, "heff_tflop_per_step": 33.1, "gpu_launches": 123456,
            "launches_per_step": 6172.8, "step_host_phases": [dict(phases)] * steps,
            "step_device_phases_ms": [dict(phases)] * steps, "step_os": [dict(phases)] * steps,
            "step_plans_built": [3] * steps, "kept": [3072] * 8, "bond_dims_block": [3072] * 6, "clocks": None,
            "heff_parts": dict(phases), "host_load": dict(phases), "energy": -47.95547901582197,
            "szsz": [-0.0849423138937656] * 3, "szsz_pairs": [[0, 1]] * 3, "dE_per_site_vs_fp64": 2.412345678901e-9,
            "szsz_max_abs_err_vs_fp64": 3.123456789012e-7, "speedup_vs_fp64": 2.1712345678,
            "full_sweep": {"seconds": 9.481234567, "energy": -47.95547933511823, "max_bond_dim": 3072,
                           "speedup_vs_fp64": 1.9312345, "dE_per_site_vs_fp64": 2.4e-9},
            "kernel_rooflines": {"L*x and *R": {"frac": 0.7012345678, "peak_source": "x" * 80},
                                 "*mid": {"frac": 0.54123456, "peak_source": "x" * 80}},
            "roofline": {"peak_source": "x" * 200}, "e2e": dict(phases)}


def test_line_is_short_and_complete():
    out = {"metric": bench.METRIC, "value": 10.71012345678901, "unit": "s/sweep", "n_gpus": 1, "steps": 200,
           "warmup": 5, "ms_per_step": 450.9512345678, "higher_is_better": False, "scaling": "weak",
           "vs_baseline": None, "dtype": "tf32x3+f64", "data": "synthetic",
           "config": {"workload": "x" * 260, "precision": "x" * 160, "l2": "x" * 100, "step": "x" * 90, "setup": "x" * 240,
                      "value_definition": "x" * 80, "ramp_energies": [-47.95547901582197] * 7, "ramp_seconds": 26.5},
           "heff_tflops": 120.1, "roofline": {"frac": 0.48123456789, "kernel": "x" * 120, "peak_source": "x" * 140},
           "cpu_baseline": None,
           "e2e": {"value": 11.0, "unit": "s/sweep", "h2d_bytes_per_step": 1, "d2h_bytes_per_step": 1},
           "gpu_launches": 123456, "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": []},
           "mixed": _arm(200), "fp64": _arm(200), "peaks_measured": {"fp64": 35.4563323726006, "tf32": 753.5856}}
    line = json.loads(json.dumps(bench.compact(out)))
    assert len(json.dumps(line)) <= 2900 and set(line) == set(out)
    for k in ("metric", "unit", "n_gpus", "steps", "warmup", "higher_is_better", "scaling", "e2e", "gpu_launches", "clocks"):
        assert line[k] == out[k], k
    assert abs(line["value"] / out["value"] - 1.0) <= 1e-6 and line["mixed"]["energy"] == out["mixed"]["energy"]
    assert line["fp64"]["full_sweep"] == out["fp64"]["full_sweep"]
