"""bench.py --impl reference where the reference's host library is neither built nor buildable: one line that says so
and a zero exit, no traceback."""
import json
import os
import subprocess
import sys

import pytest

from oracle import build_reference

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_absent_reference_prints_unavailable(tmp_path):
    if build_reference():
        pytest.skip("reference host library present")
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1", "--warmup",
                        "3"], cwd=tmp_path, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    lines = r.stdout.strip().splitlines()
    assert len(lines) == 1
    line = json.loads(lines[0])
    assert line["impl"] == "reference" and line["unavailable"]
