"""CPU test of bench.py's line: one line of at most 4 KB with every key that
identifies and qualifies the measurement, whatever the number of workloads."""
import json
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def record(bench, name, surrogate=False):
    x = 123456789.0123456789
    rec = {"metric": bench.METRIC, "value": x, "unit": "elements/s", "n_gpus": 1, "steps": 20, "warmup": 5,
           "ms_per_step": 1.23456789012345, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
           "dtype": "fp32 element math, fp64 geometry + CSR values", "data": "synthetic (seeded mesh jitter and fields)",
           "config": {"workload": name, "desc": bench.WORKLOADS[name]["desc"], "elements": 1572864,
                      "nnz": [10 ** 9] * 3, "rows": [10 ** 7] * 3, "parallelism": "1 GPU", "l2": "a" * 100,
                      "algorithmic_bytes_per_element": x, "wall_s_timed_region": x, "stages_ms_from": "b" * 60},
           "step_roofline": {"bound": "hbm", "achieved": x, "peak": x, "unit": "GB/s", "frac": 0.123456789,
                             "peak_source": "c" * 40},
           "roofline": {"bound": "hbm", "kernel": "d" * 20, "achieved": x, "peak": x, "unit": "GB/s", "frac": 0.2,
                        "traffic": 10 ** 10, "bytes_per_launch": 10 ** 10, "ms_per_launch": x, "peak_source": "e" * 40},
           "stage_rooflines": {s: {"bound": "hbm", "gbs": x, "frac": 0.1} for s in ("s1", "s2", "s3", "s4")},
           "stages_ms": {s * 12: x for s in "abcd"}, "gpu_launches": 80,
           "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": [], "samples": 3},
           "e2e": {"value": x, "unit": "elements/s", "h2d_bytes_per_step": 10 ** 8, "d2h_bytes_per_step": 10 ** 10,
                   "ms_per_step": x, "note": "f" * 200},
           "cpu_baseline": {"value": x, "unit": "elements/s", "cores": 1, "kind": "port", "sample": "g" * 300},
           "parity": {"00": 2.345678e-7, "01": 1.1e-7, "10": 1e-7, "res_u": 1.2345678e-6, "res_p": None, "rows_u": 30000,
                      "rows_p": 1000, "sample": "h" * 100, "tolerance": {"blocks": 1e-6, "residuals": 1e-5}}}
    if surrogate:
        rec["surrogate"] = {"speedup_vs_plain": 0.6712345, "stress_rel_fro": 1.234567e-4, "tangent_rel_fro": 2e-3,
                            "training": {"loss_history": [x] * 40}}
        rec["parity"] = None
    return rec


def test_line_is_short_and_complete():
    sys.path.insert(0, ROOT)
    import bench
    out = record(bench, "ns48")
    out["dirichlet"] = out["mesh_frontend"] = {"what": "i" * 300}
    out["workloads"] = {n: record(bench, n, n == "aniso64s") for n in bench.SUB_WORKLOADS}
    text = json.dumps(bench.summary(out))
    assert len(text) <= 4096 and "\n" not in text and len(json.dumps(out)) > 16384
    line = json.loads(text)
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
              "vs_baseline", "dtype", "data", "gpu_launches", "clocks"):
        assert line[k] == out[k]
    for k in ("value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"):
        assert line["e2e"][k] == out["e2e"][k]
    for k in ("workload", "elements", "parallelism", "l2"):
        assert line["config"][k] == out["config"][k]
    assert list(line["workloads"]) == bench.SUB_WORKLOADS
    assert line["workloads"]["nh64"] == {"value": 123456789, "ms_per_step": 1.2346, "frac": 0.1235, "e2e": 123456789,
                                         "parity": 1.23e-6}
    assert line["workloads"]["aniso64s"]["speedup_vs_plain"] == 0.6712 and "parity" not in line["workloads"]["aniso64s"]


def test_line_without_other_workloads():
    sys.path.insert(0, ROOT)
    import bench
    out = record(bench, "ns48")
    out["cpu_baseline"] = None
    line = bench.summary(out)
    assert "workloads" not in line and line["cpu_baseline"] is None and line["value"] == out["value"]
