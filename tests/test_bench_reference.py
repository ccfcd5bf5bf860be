"""bench.py --impl reference without a build of the reference: one line that says so."""
import json
import os
import subprocess
import sys

import pytest

from oracle.pyoracle import ref_available

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(ref_available(True), reason="the reference is built here")
@pytest.mark.parametrize("workload", [[], ["--workload", "circuit20"]])
def test_reference_arm_says_that_it_is_unavailable(workload):
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--gpus", "1",
                        "--steps", "1", "--warmup", "0"] + workload, capture_output=True, text=True, cwd=ROOT)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
