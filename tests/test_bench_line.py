"""The benchmark's one JSON line stays short enough to be read back from the end of a log, whatever
the number of timed sweeps, and keeps the run's own keys and every leg's numbers."""
import json

import bench


def _run(steps):
    sweep = {k: 0.123456789012 for k in ("sweep_s", "heff_s", "gemm_s", "svd_s", "env_s", "energy")}
    bucket = {"bucket": 3, "candidates": [None, 64, 96], "ms": [1.234567] * 3, "settled": True,
              "chosen": 64, "timed": 3}
    leg = {"workload": "w", "note": "n" * 200, "split": {**sweep, "timed_sweeps": [sweep] * steps},
           "fp64": {**sweep, "timed_sweeps": [sweep] * steps}, "dE_rel": 1e-12,
           "same_bond_dims": True, "svd_schedule": [bucket] * 30}
    base = {"metric": bench.METRIC, "value": 0.59, "unit": "s/sweep", "n_gpus": 1, "steps": steps,
            "warmup": 5, "ms_per_step": 590.0, "higher_is_better": False, "scaling": "weak",
            "vs_baseline": None, "dtype": "f64", "data": "synthetic", "config": {"model": "m"},
            "gpu_launches": 1, "roofline": {"frac": 0.1, "kernel": "k"},
            "clocks": {"sm_mhz": 2070.0, "reasons": []}, "e2e": {"value": 0.6, "what": "x"},
            "cpu_baseline": {"value": 4.5, "sample": "s"}, "svd_schedule": [bucket] * 30}
    return base, {**base, **{k: leg for k in bench.LEGS}}


def test_line_is_short_and_keeps_the_numbers():
    for steps in (1, 20, 200):
        base, res = _run(steps)
        line = bench.headline(res)
        assert len(json.dumps(line)) < 6000
        for k, v in base.items():
            if k != "svd_schedule":
                assert line[k] == v
        for leg in bench.LEGS:
            assert line[leg]["dE_rel"] == 1e-12 and line[leg]["same_bond_dims"] is True
            assert abs(line[leg]["split"]["sweep_s"] - 0.123457) < 1e-9
            assert "timed_sweeps" not in line[leg]["split"] and "svd_schedule" not in line[leg]
    assert bench.headline({"quench": {"error": "E: e"}})["quench"] == {"error": "E: e"}
