"""The octet storage of the off-diagonal blocks, on the host: steps per octet, a
place of its own for each side of each block, the other node at that place, and
valid nodes in the padding (tests/octet_layout_check.cpp).  A wrong place is a
block written outside its array, a wrong node a wrong or outside read."""

from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_octets_hold_every_block_twice(tmp_path):
    exe = tmp_path / "octet_layout_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-fopenmp", "-ffp-contract=off",
                    str(ROOT / "tests" / "octet_layout_check.cpp"), str(ROOT / "nricp_b200" / "csrc" / "host.cpp"),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0 and out.stdout.strip().endswith("ok"), out.stdout + out.stderr
