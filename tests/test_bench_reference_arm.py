"""bench.py --impl reference without the oracle's libopus (CPU only)."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_says_what_is_missing():
    from oracle.corpus import REF_LIB
    if os.path.exists(REF_LIB):
        pytest.skip("the oracle's libopus is built")
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--gpus", "1", "--steps", "1", "--warmup", "1"],
                       cwd=ROOT, capture_output=True, text=True, timeout=300)
    line = json.loads(r.stdout)
    assert r.returncode == 0 and line["impl"] == "reference" and "libopus_ref.so" in line["unavailable"], r.stderr[-2000:]
