"""Kernel attributes and occupancies are kept per device and not per process: the
holder makes its value once for every device (tests/per_device_check.cpp), and
no once-per-process initialiser of either is left in the sources."""

from __future__ import annotations

import re
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "nricp_b200" / "csrc"


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_a_value_is_made_once_per_device(tmp_path):
    exe = tmp_path / "per_device_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", str(ROOT / "tests" / "per_device_check.cpp"), "-o",
                    str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0 and out.stdout.strip().endswith("ok"), out.stdout + out.stderr


@pytest.mark.parametrize("source", sorted(p.name for p in CSRC.glob("*.cu")))
def test_nothing_of_a_device_is_initialised_once_per_process(source):
    text = (CSRC / source).read_text()
    for match in re.finditer(r"static const [\w:]+ \w+ = \[[^\]]*\]", text):
        body = text[match.start():text.index("}();", match.start())]
        assert not re.search(r"cudaFuncSetAttribute|cudaOccupancy|cudaDeviceGetAttribute", body), body
