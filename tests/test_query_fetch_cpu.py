"""The ray queries' fetch counters after refused launches, host side
(tests/cpp/query_fetch_check.cpp)."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parents[1]
SRC = REPO / "tests" / "cpp" / "query_fetch_check.cpp"


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_queries_start_from_zero(tmp_path):
    exe = tmp_path / "query_fetch_check"
    subprocess.run(["g++", "-std=c++17", "-O2", str(SRC), "-o", str(exe)], check=True)
    proc = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert proc.returncode == 0, proc.stdout + proc.stderr
