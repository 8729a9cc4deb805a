"""The window-table suites against the bounds-checked build of the library, in
which every load of the query kernels is checked before it is made: above 2^18
queries, with level 0 in DRAM, with 64-bit positions, at the largest sizes, in
every form and in batches without argmin tables."""
from __future__ import annotations

import os
import re
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]
CHECKED = ROOT / "gpu-rmq_gb300" / "librmq_gb300_checked.so"
SUITES = ["tests/test_gpu_window.py", "tests/test_gpu_window_forms.py", "tests/test_gpu_window_top.py",
          "tests/test_gpu_batch_places.py"]


def test_window_suites_under_bounds_checked_build(cuda):
    env = dict(os.environ, RMQ_GB300_LIB=str(CHECKED), RMQ_EXPECT_CHECKED_LIB="1")
    cmd = [sys.executable, "-m", "pytest", *SUITES, "-m", "gpu", "-x", "-q", "-p", "no:cacheprovider"]
    r = subprocess.run(cmd, cwd=ROOT, env=env, capture_output=True, text=True, timeout=1800)
    tail = r.stdout[-4000:] + r.stderr[-2000:]
    assert r.returncode == 0, tail
    assert "out-of-level loads 0" in r.stdout, tail
    ran = re.search(r"(\d+) passed", r.stdout)
    assert ran is not None and int(ran.group(1)) >= 170, tail  # the suites really ran
