"""bench.py without a GPU: its reference arm measures the reference's own code
or says that it cannot."""
import json
import os
import subprocess
import sys

import pytest

import oracle

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(oracle.ref_available(), reason="the reference's CUDA build is here")
def test_reference_arm_without_the_reference_is_unavailable():
    out = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1"],
                         capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stderr
    line = json.loads(out.stdout)
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
