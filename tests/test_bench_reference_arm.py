"""bench.py's reference arm where the reference was not built: one line that says
so, and success."""
import json
import os
import subprocess
import sys

import pytest

from oracle import refsim

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(refsim.available(), reason="the reference is built here: the arm runs it")
def test_missing_reference_is_reported():
    p = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--gpus", "1", "--steps", "1", "--warmup", "3"],
                       cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr
    line = json.loads(p.stdout.splitlines()[-1])
    assert line["impl"] == "reference" and "not built" in line["unavailable"]
