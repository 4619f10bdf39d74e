"""bench.py where the reference's compiled library is absent and cannot be built: its own
line comes without a CPU baseline, the reference arm's says so and exits with 0."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ABSENT = ("import sys, types, bench; from oracle import oracle as O; O.ref_available = lambda: False; "
          "O.build = lambda *a, **k: None; ")


def run(code):
    out = subprocess.run([sys.executable, "-c", ABSENT + code], cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stderr[-2000:]
    return [json.loads(line) for line in out.stdout.splitlines() if line.startswith("{")]


def test_reference_arm_says_so():
    (line,) = run("sys.argv = ['bench.py', '--impl', 'reference', '--steps', '1', '--warmup', '1']; bench.main()")
    assert line["impl"] == "reference" and line["unavailable"] and "\n" not in line["unavailable"]


def test_no_cpu_baseline():
    (line,) = run("import json; print(json.dumps({'b': bench.cpu_baseline(types.SimpleNamespace(cpu_nx=2, nx=60))}))")
    assert line["b"] is None
