"""bench.py's result line stays short: whoever runs it may keep the last 3 KB of the output only, and a longer
line is lost with everything in it."""
import json
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
import bench  # noqa: E402

CONTRACT = {"metric": bench.METRIC, "value": 18973912345.123456, "unit": "site*RHS/s", "n_gpus": 1, "steps": 20,
            "warmup": 5, "ms_per_step": 0.6633, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "f32", "data": "synthetic (seeded SU(3) links, Gaussian spinors)",
            "config": bench.workload_config(bench.L_BENCH, bench.NC, bench.NRHS, 1, "fp32"),
            "roofline": {"text": "r" * 300}, "rel_err": {"text": "e" * 240},
            "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": []}, "gpu_launches": 20,
            "e2e": {"value": 793318990.7, "unit": "site*RHS/s", "h2d_bytes_per_step": 2415919104,
                    "d2h_bytes_per_step": 2415919104, "path": "p" * 520}, "cpu_baseline": {"text": "c" * 210}}


def _full():
    solve = {"seconds": 0.0599, "seconds_cold": 0.5571, "iterations": 24, "reliable_updates": 3,
             "max_true_residual": 9.226759246474065e-11, "all_converged": True}
    return dict(CONTRACT,
                sweep=[{"precision": p, "nrhs": r, "ms": 1.0, "site_rhs_per_s": 18973912345, "gbs": 1.0, "hbm_frac": 0.5,
                        "gflops": 1.0} for p in ("fp64", "fp32", "fp16", "bf16") for r in (1, 4, 12, 24)],
                fma_peaks={"fp64_tflops": 1.26, "fp32_tflops": 76.7},
                solve={"workload": "24^3x48 SU(3) nrhs=12 kappa=0.12 point sources, tol 1e-10 (FP64 true residual)",
                       "fp32_inner": solve, "fp16_inner": solve, "fp64_plain": solve,
                       "speedup_fp32_inner_vs_fp64": 3.52, "speedup_fp16_inner_vs_fp64": 2.37},
                serve={"workload": "w" * 220, "rates": [{"rate_req_s": 5.0}] * 5, "p50_s": 0.0943, "p99_s": 0.2753,
                       "solves_per_s": 19.8, "all_ok": True, "serial_fp64_solves_per_s": 4.2},
                multi_lattice={"text": "m" * 600}, colors=[{"text": "k" * 300}] * 60)


def test_line_is_short_and_whole():
    line, tables = bench.split_line(_full())
    text = json.dumps(line)
    assert len(text) <= 2800 and "\n" not in text
    assert {k: line[k] for k in CONTRACT} == CONTRACT
    assert line["solve"]["seconds"]["fp32_inner"] == 0.0599 and line["solve"]["all_converged"]
    assert line["serve"]["p99_s"] == 0.2753
    assert tables == {k: _full()[k] for k in bench.TABLES}


def test_skipped_tables():
    line, tables = bench.split_line(dict(CONTRACT, sweep=[], solve=None, serve=None, multi_lattice=None, colors=None))
    assert tables == {} and line == CONTRACT
