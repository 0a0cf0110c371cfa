"""bench.py --impl reference where the reference's program is not built: one
line that says so, and exit code 0."""
import json
import subprocess
import sys
from pathlib import Path

import pytest

from oracle.oracle import harness_path

REPO = Path(__file__).resolve().parents[1]


def test_an_absent_reference_is_reported_as_unavailable():
    if harness_path(2, "omp3", fast=True).exists():
        pytest.skip("the reference program is built here")
    r = subprocess.run([sys.executable, str(REPO / "bench.py"), "--impl", "reference", "--gpus", "1", "--steps", "1",
                        "--warmup", "1"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout)
    assert line["impl"] == "reference" and line["unavailable"]
