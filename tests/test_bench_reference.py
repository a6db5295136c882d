"""The benchmark's reference arm: GElib cannot be built here, so the arm says so and times nothing in its place."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_the_reference_arm_says_that_the_reference_is_unavailable():
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--gpus", "1", "--steps", "1", "--warmup", "0",
                        "--workload", "cfg1"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout)
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
