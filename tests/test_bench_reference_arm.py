"""bench.py's reference arm where the reference could not be built: one line that
says so, and a clean exit."""
import json
import os
import subprocess
import sys

import pytest

import oracle
from conftest import ROOT


@pytest.mark.skipif(os.path.exists(oracle.LIB_REF_CPU), reason="the reference is built here")
def test_reference_arm_says_that_it_is_unavailable():
    p = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--lines", "100000", "--steps", "1",
                        "--warmup", "0"], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-2000:]
    line = json.loads(p.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and "libref_cpu" in line["unavailable"] and "\n" not in line["unavailable"]
