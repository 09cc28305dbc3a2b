"""bench.py's reference arm runs the unmodified reference or says in one line why not:
nothing of this repository stands in for it."""
import json
import os
import subprocess
import sys

from conftest import ROOT


def test_reference_arm():
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1"],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-1000:]
    line = json.loads(r.stdout.strip())
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
