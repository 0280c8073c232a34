"""bench.py without a GPU: its command line parses and every library
function it calls exists (the GPU runs of the benchmark cannot catch a
misspelt name before the section that uses it)."""
import os
import re
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_bench_help():
    out = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--help"], capture_output=True, text=True,
                         timeout=120)
    assert out.returncode == 0 and "--impl" in out.stdout


def test_bench_api_names_exist():
    from tokura_zgeev_batched_gb300 import api

    src = open(os.path.join(ROOT, "bench.py")).read()
    names = set(re.findall(r"\bapi\.([A-Za-z_]\w*)", src))
    assert names and not [n for n in names if not hasattr(api, n)]
    lib = api.lib()
    syms = set(re.findall(r"\bapi\.lib\(\)\.([A-Za-z_]\w*)", src))
    assert not [s for s in syms if not hasattr(lib, s)]


def test_reference_arm_json_line():
    """`bench.py --impl reference` (the LAPACK CPU path) prints one JSON line with the
    contract's keys; it needs no GPU."""
    import json

    out = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1",
                          "--warmup", "1"], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stderr[-2000:]
    lines = [ln for ln in out.stdout.splitlines() if ln.startswith("{")]
    assert len(lines) == 1
    d = json.loads(lines[0])
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better",
                "scaling", "vs_baseline", "dtype", "data", "config", "cpu_baseline", "e2e"):
        assert key in d, key
    assert d["impl"] == "reference" and d["value"] > 0 and d["higher_is_better"] is True
    assert d["cpu_baseline"]["value"] == d["value"] and d["cpu_baseline"]["cores"] >= 1
    assert d["e2e"]["h2d_bytes_per_step"] == 0 and d["e2e"]["d2h_bytes_per_step"] == 0


def test_clock_record_summary():
    """The `clocks` object of the JSON line: median SM clock, max clock and power, and the
    throttle reasons seen Active during the timed region (nvidia-smi csv, noheader, nounits)."""
    sys.path.insert(0, ROOT)
    import bench

    lines = [
        "2070, 2070, 612.5, 0x0000000000000000, Not Active, Not Active, Not Active, Not Active",
        "2055, 2070, 640.1, 0x0000000000000004, Not Active, Not Active, Not Active, Active",
        "1980, 2070, 655.0, 0x0000000000000004, Not Active, Not Active, Not Active, Active",
        "garbage line",
        "[N/A], 2070, 600.0, 0x0, Not Active, Not Active, Not Active, Not Active",
    ]
    s = bench.ClockSampler.summarize(lines)
    assert s["sm_mhz"] == 2055 and s["sm_max_mhz"] == 2070 and s["samples"] == 3
    assert s["power_w_max"] == 655.0 and s["reasons"] == ["sw_power_cap"]
    hot = bench.ClockSampler.summarize(["1500, 2070, 700, 0x8, Not Active, Active, Not Active, Not Active"])
    assert hot["reasons"] == ["hw_thermal_slowdown"]
    assert bench.ClockSampler.summarize([]) is None


def test_the_line_is_short_and_keeps_the_contract():
    """Long records (every configuration with its details) are cut to a line that a log's tail holds."""
    import json

    sys.path.insert(0, ROOT)
    import bench

    long = {"value": 1.23456789e5, "note": "x" * 2000, "inner": {"a": [1.5] * 200}, "flags": [0] * 500}
    out = {"metric": bench.METRIC, "value": 189000.123456, "unit": "matrices/s", "n_gpus": 1, "steps": 20, "warmup": 5,
           "ms_per_step": 346.1234567, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
           "dtype": "c128 (f64)", "data": "synthetic", "gpu_launches": 60, "flagged": 0,
           "config": {"workload": "w" * 150, "n": 64, "global_batch": 65536, "l2": "l" * 60, "arithmetic": "a" * 200},
           "roofline": {"bound": "b" * 70, "achieved": 1.9, "peak": 1.2, "unit": "TFLOP/s", "frac": 1.5,
                        "int_mad": {"peak": 6.7, "unit": "TFLOP/s", "frac": 0.3, "peak_source": "p" * 90}},
           "cpu_baseline": {"value": 9000.0, "unit": "matrices/s", "cores": 16, "kind": "port", "sample": "s" * 400},
           "e2e": {"value": 184000.5, "unit": "matrices/s", "h2d_bytes_per_step": 4 << 30, "d2h_bytes_per_step": 1 << 26,
                   "host_buffers": long},
           "clocks": {"sm_mhz": 2070, "sm_max_mhz": 2070, "reasons": ["sw_power_cap"], "power_w_max": 600.0, "samples": 40},
           "parity": dict(long, max_rel_err_fro=1e-15, flag_mismatch=0)}
    for k in range(12):
        out[f"configuration_{k}"] = dict(long, **{f"field_{i}": i * 1.1 for i in range(20)})
    text = bench.short_line(out)
    assert len(text) <= bench.LINE_BYTES and "\n" not in text
    d = json.loads(text)
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
                "vs_baseline", "dtype", "data", "config", "cpu_baseline", "e2e", "clocks", "gpu_launches"):
        assert key in d, key
    assert d["value"] == out["value"] and d["clocks"]["reasons"] == ["sw_power_cap"] and d["config"]["n"] == 64
    assert set(d["e2e"]) == {"value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"}
