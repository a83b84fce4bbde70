"""The smoke entry point, with or without the oracle's libopus."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.gpu
def test_smoke_entry_point(cuda):
    r = subprocess.run([sys.executable, "__graft_entry__.py", "smoke"], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "bit-exact" in r.stdout, (r.stdout + r.stderr)[-2000:]
