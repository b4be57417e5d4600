"""CPU: the bench's reference arm where the reference's CPU library is not
built: one JSON line that says so, and exit code 0."""
import json
import os
import subprocess
import sys

import pytest

import gasref
from conftest import ROOT


def test_reference_arm_says_it_is_unavailable():
    if gasref.available():
        pytest.skip("the reference library is built here")
    run = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--gpus", "1",
                          "--steps", "1", "--warmup", "3"], capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert run.returncode == 0, run.stderr[-2000:]
    line = json.loads(run.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"]
