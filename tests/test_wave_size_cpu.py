"""Wave sizes within the shadow list's slots and counts, host side
(tests/cpp/wave_size_check.cpp)."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parents[1]
SRC = REPO / "tests" / "cpp" / "wave_size_check.cpp"


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_waves_fit_their_counters(tmp_path):
    exe = tmp_path / "wave_size_check"
    subprocess.run(["g++", "-std=c++17", "-O2", str(SRC), "-o", str(exe)], check=True)
    proc = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert proc.returncode == 0, proc.stdout + proc.stderr
