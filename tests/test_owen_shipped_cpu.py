"""The Owen-scrambled dimensions with the tables the library makes, host side
(tests/cpp/owen_shipped_check.cpp)."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parents[1]
SRC = REPO / "tests" / "cpp" / "owen_shipped_check.cpp"


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_shipped_owen_values_equal_every_digit(tmp_path):
    exe = tmp_path / "owen_shipped_check"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", str(SRC), "-o", str(exe)], check=True)
    proc = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert proc.returncode == 0, proc.stdout + proc.stderr
