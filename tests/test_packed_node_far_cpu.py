"""The traversal's packed BVH nodes (pt_node.cuh) far from the world's origin, host
side (tests/cpp/packed_node_far_check.cpp)."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parents[1]
SRC = REPO / "tests" / "cpp" / "packed_node_far_check.cpp"


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_far_packed_boxes_hold_the_boxes(tmp_path):
    exe = tmp_path / "packed_node_far_check"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", str(SRC), "-o", str(exe)], check=True)
    proc = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert proc.returncode == 0, proc.stdout + proc.stderr
