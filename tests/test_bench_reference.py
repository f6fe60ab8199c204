"""bench.py's reference arm is the Arm NN runtime or nothing: no stand-in of this repository is timed in its name."""
import json
import os
import subprocess
import sys

import pytest

from armnn_b200 import armnn_host

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(armnn_host.available(), reason="the Arm NN runtime is built here")
def test_reference_arm_without_the_runtime_says_so():
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--steps", "1", "--warmup", "0"], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
