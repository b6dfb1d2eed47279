"""The line bench.py prints: readers keep only the end of a run's output, so a whole run's line has to stay short, with every
key of the headline in it."""
import json

import bench

CLOCKS = {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": ["sw_power_cap", "hw_thermal_slowdown"], "samples": 600,
          "interval_ms": 1000}
X = 123456789.123456789
TEXT = "what was measured, and how, " * 20


def _full():
    seg = {k: X / 1e8 for k in ("kdp", "sort", "tree", "nbr_prep", "dens_list", "dens", "eos", "drvt_list", "drvt",
                                "hydro_list", "hydro", "grav_list", "grav", "final", "entropy")}
    errors = {f: {q: 1.23456789e-7 for q in ("p50", "p99", "p99.9", "max", "l2_rel")} for f in "abcdefgh"}
    part = {"value": X, "unit": "particle-steps/s", "s_per_step": 0.123456789, "vs_cpu_baseline": 300.123456789, "config": TEXT}
    latency = {"step_latency_s": {"p50": 0.0123456789, "p99": 0.0223456789}}
    out = {"metric": bench.METRIC, "value": X, "unit": "particle-steps/s", "n_gpus": 1, "steps": 20, "warmup": 5,
           "ms_per_step": 6.390123456789, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
           "dtype": "f32 pair sums + f64", "data": "synthetic (seeded IC generator, synthetic 200x200 rho-u tables)",
           "config": {"workload": "1,000,000-particle two-layer impact (90% target, 10% impactor, iron/dunite, 30 deg, "
                                  "1.2 v_esc), theta 0.5", "particles": 1000000, "precision": "mixed",
                      "l2": "inputs larger than L2 (no flush)", "parallelism": "1 GPU"},
           "gpu_launches": 12345, "clocks": CLOCKS,
           "roofline": {"bound": "fp32", "kernel": "gravity", "achieved": X, "peak": X, "unit": "TFLOP/s", "frac": 0.123456789,
                        "work_per_launch": X, "ms_per_launch": 1.23456789, "traffic": None, "peak_source": TEXT},
           "rooflines": {k: {"achieved": X, "note": TEXT} for k in seg}, "segments_ms_per_step": seg,
           "segment_share": seg, "work": {k: 123456789 for k in seg}, "peaks": {"hbm_gbs": 6791.4}, "autotune": {"x": TEXT},
           "drift": {"mixed": errors}, "e2e": {"value": X, "unit": "particle-steps/s", "h2d_bytes_per_step": 123456789,
                                               "d2h_bytes_per_step": 123456789, "steps": 5},
           "fp64": {"value": X, "ms_per_step": 140.123456789, "segments_ms_per_step": seg, "clocks": CLOCKS, "roofline": {}},
           "multiwalk": {**part, "index_form": part, "host_staging": part, "fp64": part},
           "mixed_error_vs_fp64": errors,
           "config_4m": {"workload": TEXT, **{f"theta_{t}": {p: {"ms_per_step": 25.123456789, "value": X, "drift": errors}
                                                            for p in ("mixed", "fp64")} for t in (0.5, 0.7)}},
           "batch": {**part, **latency}, "serving": {**part, **latency, "clocks": CLOCKS},
           "cpu_baseline": {"value": X, "unit": "particle-steps/s", "cores": 16, "kind": "port",
                            "sample": "oracle restatement (OpenMP) on the same workload (1000000 particles), 5 steps after "
                                      "the prologue (11.6 s on 16 threads)"}}
    return out


def test_the_line_of_a_whole_run_is_short_and_complete():
    out = _full()
    line = json.loads(json.dumps(bench.result_line(out)))
    assert len(json.dumps(line)) < bench.LINE_MAX
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
              "vs_baseline", "dtype", "data", "config", "gpu_launches", "clocks", "e2e"):
        assert line[k] == out[k]
    assert line["multiwalk"]["index_form"] and line["config_4m"]["theta_0.7"]["fp64"] and line["serving"]["value"]


def test_a_run_without_the_other_sections():
    out = {k: v for k, v in _full().items() if k not in ("fp64", "multiwalk", "config_4m", "batch", "serving", "cpu_baseline",
                                                        "e2e", "mixed_error_vs_fp64")}
    assert bench.result_line(out)["value"] == out["value"]
