"""The line bench.py prints: every key its readers take from it, in a few kilobytes however
many solves were timed (--full has the rest)."""
import json

import bench


def _line(solves):
    clocks = {"sm_mhz": 2024.5, "sm_max_mhz": 2070.0, "reasons": ["sw_power_cap"], "samples": 10}
    est = [1.0751456065903934e-10 * (i + 1) for i in range(solves)]
    acc = {"err_vs_fp64_max": 1.063023558067755e-08, "err_vs_fp64": est[:4], "err_est_same_solves": est[:4],
           "solves_checked": 4, "note": "n" * 100}
    fp64 = {"value": 0.29723774266221537, "unit": "solves/s", "steps": 4, "ms_per_step": 3364.310302734375, "lanes": 4,
            "note": "n" * 100}
    fact = {"complex64": solves, "fp64class": 0, "fp64_fallback": 0}
    sub = {"value": 357.8406860965593, "unit": "solves/s", "ms_per_step": 2.7945396900177, "steps": solves,
           "config": {"workload": "w" * 400, "N": "1536-15516"}, "err_est": est, "factorization": fact, "serving": None,
           "fp64_path": fp64, "accuracy": acc, "mixed_over_fp64": 7.0290760743677945, "clocks": clocks, "cmd": "c" * 100}
    roof = {"bound": "tensor", "achieved": 155.91482302529877, "peak": 1714.7, "unit": "TFLOP/s",
            "frac": 0.0909283390828126, "avg_launch_ms": 3.486553624678742, "launches": 55, "traffic": 3300612207.7090907,
            "executed_frac": 0.7880114035005433, "ms_share": 0.404153577482994}
    return {"metric": bench.METRIC, "value": 10.072345804090906, "unit": "solves/s", "n_gpus": 1, "steps": solves,
            "warmup": 5, "ms_per_step": 99.28173828125, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "c64+c128", "data": "synthetic (seeded generated meshes; no dataset)",
            "config": {"workload": "w" * 130, "precision": "mixed", "N": 7680, "parallelism": "replicas x1", "lanes": 4,
                       "batch": 1, "solver": "escalate", "l2": "l" * 45},
            "err_est": est, "refine_iters": [2] * solves, "factorization": fact, "gpu_launches": 22255,
            "tiles": {"near_minb": 4, "far_rows": 4, "raster": 4, "source": "tuned", "seconds": 4.047443168000001},
            "clocks": clocks, "P_sample": est[:2], "fp64_path": fp64, "mixed_over_fp64": 33.886496761406384, "accuracy": acc,
            "serving": {"arrivals": "poisson", "rate_per_s": 8.057876643272726, "requests": 64, "solves_per_request": 1.0,
                        "p50_ms": 322.112016, "p99_ms": 590.4735721599999, "mean_ms": 313.434085,
                        "solves_per_s": 8.086145099930507, "lanes": 4},
            "e2e": {"value": 10.106018929818513, "unit": "solves/s", "h2d_bytes_per_step": 184416, "d2h_bytes_per_step": 28,
                    "clocks": clocks},
            "stage_ms": {k: 11.453904151916504 for k in ("ms_fill", "ms_lu", "ms_solve", "ms_trace", "ms_refine")},
            "kernel_ms_per_step": {k: 5.028640031814575 for k in ("fill_far", "fill_near", "gather", "lu_panel", "lu_gemm",
                                                                  "trsm", "solve_gemm", "trace", "refine_gemm", "slice")},
            "kernel_ms_note": "n" * 100, "roofline": {**roof, "kernel": "ex_gemm", "kinds": ["refine_gemm", "trace"],
                                                      "peak_source": "measured bf16 sustained", "note": "n" * 150},
            "rooflines": {g: roof for g in ("ex_gemm", "tc_gemm", "lu_panel", "fill", "memory")},
            "subs": {nm: sub for nm in ("cube4", "tip", "slab", "mix")},
            "cpu_baseline": {"value": 0.04285564610103604, "unit": "solves/s", "cores": 16, "kind": "port",
                             "sample": "s" * 360, "spread": {"min": 0.0427, "median": 0.0428, "max": 0.0429, "steps": 3}}}


def test_line_keeps_its_keys_and_stays_short():
    full = _line(256)
    text = json.dumps(bench.compact(full))
    assert len(text) < 3000, len(text)
    d = json.loads(text)
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
              "vs_baseline", "dtype", "data", "config", "clocks", "e2e", "gpu_launches", "roofline"):
        assert k in d, k
    assert d["value"] == full["value"] and d["ms_per_step"] == full["ms_per_step"]
    assert d["clocks"] == full["clocks"] and d["config"] == full["config"]
    for k in ("value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"):
        assert d["e2e"][k] == full["e2e"][k], k
    assert d["err_est_max"] == float(f"{max(full['err_est']):.4g}")


def test_length_does_not_grow_with_the_solves():
    assert abs(len(json.dumps(bench.compact(_line(4096)))) - len(json.dumps(bench.compact(_line(16))))) < 40
