"""The benchmark's reference arm runs on the host cores (no GPU): its one JSON line must carry the keys the contract
names, and the workload table must be self-consistent."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_prints_one_contract_line():
    res = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1", "--warmup", "0"],
                         capture_output=True, text=True, timeout=600, cwd=ROOT)
    assert res.returncode == 0, res.stderr[-2000:]
    lines = [l for l in res.stdout.splitlines() if l.startswith("{")]
    assert len(lines) == 1
    d = json.loads(lines[0])
    for key in ("impl", "metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
                "vs_baseline", "dtype", "data", "config", "cpu_baseline", "e2e"):
        assert key in d, key
    assert d["impl"] == "reference" and d["unit"] == "GB/s" and d["value"] > 0 and d["steps"] == 1
    assert d["vs_baseline"] is None and d["data"] == "synthetic" and "workload" in d["config"]
    assert d["cpu_baseline"]["kind"] == "port" and d["cpu_baseline"]["cores"] >= 1 and d["cpu_baseline"]["sample"]
    assert d["e2e"]["h2d_bytes_per_step"] == 0 and d["e2e"]["d2h_bytes_per_step"] == 0 and d["e2e"]["value"] == d["value"]
    # the other configurations ride along, each with its own CPU value
    assert set(d["workloads"]) == {"c1", "c3", "c4", "c5", "meta", "fused", "next"}
    for rec in d["workloads"].values():
        assert rec["value"] > 0 and rec["unit"] in ("GB/s", "TFLOP/s") and rec["kind"] == "port" and rec["sample"]


def test_workload_tables_are_consistent():
    sys.path.insert(0, ROOT)
    import bench
    assert set(bench.WORKLOADS) == {"c1", "c2", "c3", "c4", "c5", "meta", "fused", "next"}
    assert bench.HEADLINE == "c2" and set(bench.CONFIGS) == {"c1", "c3", "c4", "c5", "meta", "fused", "next"}
    for key, cls in bench.WORKLOADS.items():
        wl = cls()
        parts = set(wl.work())
        assert parts == set(wl.launches) == set(wl.kernel_of), key
        assert set(getattr(wl, "traffic", {})) <= parts
        assert set(getattr(wl, "all_reduced", ())) <= parts
        assert wl.unit in ("GB/s", "TFLOP/s") and wl.bound in ("hbm", "tensor") and wl.scaling in ("weak", "strong")


def test_the_line_of_a_default_run_is_short_and_complete():
    """Built from records as measure() makes them, with every number at full length."""
    sys.path.insert(0, ROOT)
    import bench
    x = 1234.5678901234567
    clocks = {"sm_mhz": x, "sm_max_mhz": x, "reasons": ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"], "samples": 999,
              "window": "timed region and untimed repeats of the same step"}

    def record(key):
        wl = bench.WORKLOADS[key]
        kernel = max(wl().kernel_of.values(), key=len)
        return {"metric": wl.metric, "value": x, "unit": wl.unit, "n_gpus": 8, "steps": 50, "warmup": 5, "ms_per_step": x, "higher_is_better": True,
                "scaling": wl.scaling, "vs_baseline": None, "dtype": wl.dtype, "data": "synthetic",
                "config": {"workload": wl.description, "algorithmic_work_per_step": 10 ** 13, "l2": "no flush: " + "x" * 70, "parallelism": "dp8"},
                "clocks": clocks, "e2e": {"value": x, "unit": wl.unit, "ms_per_step": x, "h2d_bytes_per_step": 10 ** 10, "d2h_bytes_per_step": 10 ** 10},
                "gpu_launches": 10 ** 4, "collective": "peer-kernel (NVLink loads/stores, one launch per rank)", "collective_overlap": True,
                "roofline": {"bound": wl.bound, "kernel": kernel, "parts": list(wl().work()), "achieved": x, "peak": x, "unit": wl.unit, "frac": x,
                             "peak_source": "measured (burst)", "traffic": x, "step_frac": x, "note": "n" * 400},
                "parts": [{"part": p, "ms": x} for p in wl().work()], "stability": {"repetitions": 300, "ms_median": x}, "cuda_graph": True,
                "parts_timing": "p" * 60, "device_status": 0, "parity_ok": True,
                "cpu_baseline": {"value": x, "unit": wl.unit, "cores": 128, "kind": "port", "sample": "s" * 150}}
    full = dict(record(bench.HEADLINE), workloads={k: record(k) for k in bench.CONFIGS}, gpu_launches_all_workloads=10 ** 5)
    line = json.dumps(bench.contract_line(full))
    assert len(line) < 2900
    d = json.loads(line)
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling", "vs_baseline", "dtype", "data",
                "config", "clocks", "e2e", "gpu_launches", "roofline", "cpu_baseline", "parity_ok", "device_status"):
        assert key in d, key
    assert set(d["workloads"]) == set(bench.CONFIGS) and all(r["ok"] and r["value"] > 0 for r in d["workloads"].values())
    assert set(d["clocks"]) >= {"sm_mhz", "sm_max_mhz", "reasons"} and set(d["e2e"]) >= {"value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"}
