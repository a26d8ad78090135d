"""The tables of first Owen-scrambled digits (pt_common.cuh), host side
(tests/cpp/owen_table_check.cpp): the same values with and without them."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parents[1]
SRC = REPO / "tests" / "cpp" / "owen_table_check.cpp"


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_owen_tables_change_no_value(tmp_path):
    exe = tmp_path / "owen_table_check"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", str(SRC), "-o", str(exe)], check=True)
    proc = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert proc.returncode == 0, proc.stdout + proc.stderr
