"""bench.py's reference arm where the reference library is not built: one JSON
line that says so, and a normal exit."""
import json
import os
import subprocess
import sys

import pytest

from oracle import ref

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(ref.available(fast=True), reason="the reference library is here")
def test_reference_arm_says_it_is_unavailable():
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--boxes", "2", "--steps",
                        "1", "--warmup", "1"], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"]
