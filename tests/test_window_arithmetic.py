"""The index arithmetic of window-table queries at the top of the 32-bit range
(host side of gpu-rmq_gb300/csrc/rmq_window.cuh, CPU): which part of a query
windows serve, and which two windows cover it, computed with 32-bit positions
over the largest array they serve, equal the same with 64-bit positions, for
every query in the last 4096 entries and for random ones anywhere; and the
cover holds the query."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path_factory.mktemp("window") / "window_harness"
    subprocess.run([nvcc, "-O2", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "--expt-relaxed-constexpr",
                    "-I", str(ROOT / "gpu-rmq_gb300" / "csrc"), str(ROOT / "tests" / "window_harness.cu"), "-o",
                    str(exe)], check=True)
    return exe


@pytest.mark.parametrize("form", range(6))
def test_positions_near_2_pow_32(harness, form):
    out = subprocess.run([str(harness), str(form)], capture_output=True, text=True, check=True).stdout
    checked, wrong = out.split()[-3], out.split()[-1]
    assert int(checked) > 8_000_000 and wrong == "0", out
