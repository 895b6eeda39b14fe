"""The bench's reference arm times the reference's own code or says that it cannot.

Where the reference's sources were not present when oracle/_ref was built, there
is nothing of its own to time: one line says so and the exit status is 0. The
oracle's C restatement, which is this repository's code, must not stand in.
"""
import json
import subprocess
import sys

import pytest

from conftest import ROOT
from oracle import oracle


def test_reference_arm_without_the_reference():
    if oracle.ref_available():
        pytest.skip("the reference is built here")
    r = subprocess.run([sys.executable, str(ROOT / "bench.py"), "--impl", "reference", "--workload", "duct", "--steps", "1",
                        "--warmup", "3"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"]
    assert "value" not in line
