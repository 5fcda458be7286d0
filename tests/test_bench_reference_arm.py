"""bench.py's reference arm runs the reference's own CPU join (oracle/_ref) on the workload's own
inputs, generated by the oracle's restatement of the generator: it must load no engine library and
report the same `config` object as the engine's arm. Where oracle/_ref is not built it says so and runs
nothing in its place."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = r"""
import io, json, sys, contextlib
sys.argv = ["bench.py", "--impl", "reference", "--workload", "c0", "--rows", "200000", "--steps", "2",
            "--warmup", "1"]
import bench
from oracle import oracle
if PATCH:
    oracle.ref_available = lambda: False
buf = io.StringIO()
with contextlib.redirect_stdout(buf):
    bench.main()
maps = open("/proc/self/maps").read()
print(json.dumps({"line": buf.getvalue(), "engine_loaded": "libbrigjoin" in maps,
                  "modules": sorted(m for m in sys.modules if m.startswith("brig"))}))
"""


def _arm(patch):
    out = subprocess.run([sys.executable, "-c", SCRIPT.replace("PATCH", str(patch))], cwd=ROOT, capture_output=True,
                         text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    res = json.loads(out.stdout.strip().splitlines()[-1])
    assert not res["engine_loaded"] and res["modules"] == []
    line = json.loads(res["line"].strip().splitlines()[-1])
    assert line["impl"] == "reference"
    return line


def test_reference_arm_is_unavailable_without_the_reference():
    assert set(_arm(True)) == {"impl", "unavailable"}


def test_reference_arm_loads_no_engine_library(oracle):
    if not oracle.ref_available():
        pytest.skip("oracle/_ref is not built")
    line = _arm(False)
    assert line["steps"] == 2 and line["warmup"] == 1
    assert line["value"] > 0 and line["cpu_baseline"]["kind"] == "reference"
    sys.path.insert(0, ROOT)
    import bench
    wl = dict(bench.WORKLOADS["c0"])
    wl["n_r"] = wl["n_s"] = 200000
    wl["name"] = line["config"]["workload"]
    assert line["config"] == bench.workload_config(wl, 1)
