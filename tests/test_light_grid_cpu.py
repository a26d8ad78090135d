"""The light sample grid's arithmetic of pt_common.cuh, host side
(tests/cpp/light_grid_check.cpp): div_small equals the hardware quotient for
every stratified offset a grid of up to 16 strata draws (stratum + k / 2^24,
rounded), idiv_small the whole quotient for every pair."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parents[1]
SRC = REPO / "tests" / "cpp" / "light_grid_check.cpp"


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_light_grid_matches_division(tmp_path):
    exe = tmp_path / "light_grid_check"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", str(SRC), "-o", str(exe)], check=True)
    proc = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert proc.returncode == 0, proc.stdout + proc.stderr
    lines = proc.stdout.strip().split("\n")
    assert len(lines) == 2 and all(" 0 mismatches" in ln for ln in lines), proc.stdout
