"""The partition of a tile plan, kept for the plan in the other arithmetic."""
from __future__ import annotations

import subprocess
from pathlib import Path

REPO = Path(__file__).resolve().parents[1]


def test_plans_with_a_kept_partition(tmp_path):
    exe = tmp_path / "tile_partition_check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-pthread", "-I", str(REPO / "t-flows_gb300" / "csrc"),
                    str(REPO / "tests" / "native" / "tile_partition_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout
