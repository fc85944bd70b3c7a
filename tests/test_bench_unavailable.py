"""bench.py's reference arm where the reference's library is not built: one line that says so, exit code 0."""
import json
import os
import subprocess
import sys

import pytest

from oracle import oracle
from tests.conftest import ROOT


@pytest.mark.skipif(oracle.have_ref(), reason="the reference's library is built here")
def test_reference_arm_says_that_it_is_unavailable():
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1",
                        "--warmup", "3"], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    lines = [json.loads(x) for x in r.stdout.splitlines() if x.startswith("{")]
    assert len(lines) == 1 and lines[0]["impl"] == "reference" and lines[0]["unavailable"]
