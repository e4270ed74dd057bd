"""out_of_memory_cases.py in a process of its own: it takes nearly all of the device's memory,
which a failing case would keep from the tests after it, and what the driver holds back of
memory freed by the tests before it would decide how much is left."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def test_calls_that_run_out_of_memory():
    res = subprocess.run([sys.executable, "-m", "pytest", "-q", "-p", "no:cacheprovider",
                          os.path.join(HERE, "out_of_memory_cases.py")],
                         cwd=os.path.dirname(HERE), capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stdout[-4000:] + res.stderr[-1000:]
    assert "10 passed" in res.stdout
