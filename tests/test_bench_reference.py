"""bench.py's reference arm without a built reference: one JSON line that says so, and a
successful exit."""
import json
import os
import subprocess
import sys

import pytest

from conftest import ROOT


def test_reference_arm_without_its_build():
    from ftoracle import REF_DRIVER_SO
    if os.path.exists(REF_DRIVER_SO):
        pytest.skip("the reference is built here")
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1"],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"]
