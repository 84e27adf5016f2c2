"""What calls take of the device's memory, and what they do when little is left. Each case runs in a process of its own:
the library keeps its buffers for the life of the process."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
WORKER = os.path.join(os.path.dirname(os.path.abspath(__file__)), "memory_worker.py")


@pytest.mark.parametrize("case", ["velocity", "step", "copies", "far", "short", "blocks"])
def test_memory(case):
    r = subprocess.run([sys.executable, WORKER, case], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "OK" in r.stdout, (r.stdout[-2000:], r.stderr[-3000:])
