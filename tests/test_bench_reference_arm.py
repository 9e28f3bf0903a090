"""bench.py --impl reference times the reference's own build or says that there is none."""
import json
import os
import subprocess
import sys

import pytest

from conftest import ROOT


def test_reference_arm_without_the_reference():
    """Without a build of the reference the arm prints one `unavailable` line and succeeds: no other implementation's
    number stands in for the reference's."""
    from oracle.oracle import REF_SO
    if os.path.exists(REF_SO):
        pytest.skip("the reference build is present")
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1", "--warmup", "0"],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
