"""bench.py --impl reference runs the reference program or nothing: without its build the arm says
that it is unavailable, and no other code stands in for it."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_unavailable_without_the_reference(tmp_path):
    code = ("import bench, sys; bench.reference_binary = lambda: None; "
            "sys.argv = ['bench.py', '--impl', 'reference', '--steps', '2', '--warmup', '3']; sys.exit(bench.main())")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-500:]
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"]
    assert "value" not in line
