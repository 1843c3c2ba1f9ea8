"""The linear solve's shared memory over every graph size: a cluster's arrays
never exceed what its launch has, and the whole device's solve is declined where
its CTAs' arrays would (tests/solve_layout_check.cpp, on the host)."""

from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_the_solves_arrays_fit(tmp_path):
    exe = tmp_path / "solve_layout_check"
    subprocess.run(["g++", "-O2", "-std=c++17", str(ROOT / "tests" / "solve_layout_check.cpp"), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0 and out.stdout.strip().endswith("ok"), out.stdout + out.stderr
