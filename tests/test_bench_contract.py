"""The bench's reference arm on the CPU (no GPU): one JSON line with the
contract's keys, the same metric and unit as the product arm, a bounded
sample of the workload, and no work on ranks other than 0."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ARGS = ["--impl", "reference", "--grid", "16", "--particles", "1024", "--steps", "3", "--warmup", "3",
        "--cpu-seconds", "0.5"]


def _run(env_extra=None):
    env = dict(os.environ, **(env_extra or {}))
    return subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), *ARGS], cwd=ROOT, env=env,
                          capture_output=True, text=True, timeout=600)


def test_reference_arm_line():
    r = _run()
    assert r.returncode == 0, r.stderr[-2000:]
    lines = [l for l in r.stdout.splitlines() if l.startswith("{")]
    assert len(lines) == 1
    d = json.loads(lines[0])
    sys.path.insert(0, ROOT)
    import bench

    assert d["impl"] == "reference" and d["metric"] == bench.METRIC and d["unit"] == bench.UNIT
    assert d["higher_is_better"] is True and d["steps"] == 3 and d["warmup"] == 3 and d["value"] > 0
    cb = d["cpu_baseline"]
    assert cb["kind"] == "port" and cb["cores"] >= 1 and cb["value"] == d["value"]
    assert cb["sample"].startswith("1024 of 1024 particles")
    assert d["e2e"] == {"value": d["value"], "unit": d["unit"], "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}


def test_reference_arm_other_ranks_exit_without_work():
    r = _run({"WORLD_SIZE": "2", "RANK": "1", "LOCAL_RANK": "1"})
    assert r.returncode == 0 and not [l for l in r.stdout.splitlines() if l.startswith("{")]


def test_printed_line_is_compact():
    """The printed line keeps the contract's keys as they are and stays short however long the legs get."""
    sys.path.insert(0, ROOT)
    import bench

    contract = {"metric": bench.METRIC, "value": 5.5491234567e10, "unit": bench.UNIT, "ms_per_step": 19.3512345678,
                "config": {"workload": "w" * 150}, "roofline": {"kernel": "k", "frac": 0.123456789},
                "e2e": {"value": 1.23456789e10, "unit": "u", "h2d_bytes_per_step": 7}, "clocks": {"reasons": []},
                "job_latency": {"p50_s": 0.123456789}, "gpu_launches": 100}
    per_case = {f"mode{i}/{e}GeV": {f"form{f}": {f"product{q}": 0.123456789 for q in range(3)} for f in range(9)}
                for i in range(4) for e in (1, 10, 100)}
    leg = {"value": 1.23456789e11, "unit": "u" * 40, "note": "n" * 400, "roofline": {"frac": 0.87654321, "note": "x" * 80},
           "per_campaign": [{"n": 1}] * 50}
    line = dict(contract, **{k: leg for k in bench.LEGS[:-1]},
                precision={"max_rel_err_resolved": {"f32": {"D_mumu": 0.001234567}}, "within_tolerance": True,
                           "per_case": per_case, "criterion": "c" * 500})
    assert len(json.dumps(line)) > 12000
    out = bench.compact(line)
    assert len(json.dumps(out)) < 3000
    for k, v in contract.items():
        assert out[k] == v, k
    assert out["lag_pairs"] == {"value": 1.2346e11, "roofline": {"frac": 0.87654}}
    assert out["precision"] == {"max_rel_err_resolved": {"f32": {"D_mumu": 0.0012346}}, "within_tolerance": True}
    assert bench.compact(dict(contract, serving=None))["serving"] is None
