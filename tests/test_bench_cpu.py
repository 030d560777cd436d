"""The benchmark's reference arm where the reference was never compiled."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_without_the_reference():
    """It times the reference's own code or nothing: the repository's restatement must not appear under its name."""
    code = ("import sys, oracle; oracle.have_ref = lambda: False; import bench; "
            "sys.argv = ['bench.py', '--impl', 'reference', '--steps', '1', '--warmup', '0', '--workload', 'c0']; bench.main()")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout)
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
