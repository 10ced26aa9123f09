"""The benchmark's reference arm where the reference's own code was not built: one JSON line that says so
and exit status 0, with no GPU needed for it."""
import json
import os
import subprocess
import sys

import pytest

from oracle.oracle import Reference

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(Reference.available("avx2") or Reference.available("avx512"), reason="oracle/_ref is built")
def test_reference_arm_reports_a_missing_reference():
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--gpus", "1", "--steps", "2"], cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"]
