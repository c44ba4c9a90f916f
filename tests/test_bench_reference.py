"""The benchmark's reference arm without a reference library: one line that says
so, and a clean exit."""

import json
import pathlib
import subprocess
import sys

ROOT = pathlib.Path(__file__).resolve().parent.parent


def test_missing_reference_is_one_line():
    code = "import pathlib, sys; from oracle import oracle; oracle.REF_LIB_PATH = pathlib.Path('/nowhere/lib.so'); sys.argv = ['bench.py', '--impl', 'reference', '--steps', '20', '--warmup', '5']; import bench; bench.main()"
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout.splitlines()[-1])
    assert line["impl"] == "reference" and set(line) == {"impl", "unavailable"}
    assert "\n" not in line["unavailable"]
