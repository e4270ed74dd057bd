"""bench.py --skin 0 searches at every step, also where a handle without a skin would step on
lists of the library's own: six kernels a step (two on lists)."""
from __future__ import annotations

import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_skin_zero_searches_every_step():
    res = subprocess.run(
        [sys.executable, "bench.py", "--skin", "0", "--grains", "4096", "--steps", "60", "--warmup",
         "60", "--no-extras", "--no-cpu-baseline"],
        cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stderr[-2000:]
    line = [json.loads(x) for x in res.stdout.splitlines() if x.startswith("{")][-1]
    assert line["neighbor_lists"] is None
    assert line["gpu_launches"] >= 6 * 60
    assert "k_force (" in line["roofline"]["kernel"]
