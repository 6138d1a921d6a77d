"""The column-march planner (segmentctscans_b200/csrc/march_plan.cuh) chooses what its definition says, on
random masks, shapes and slots, and takes little host time (tests/cpp/march_check.cpp)."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_plans_follow_the_definition(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    exe = tmp_path / "march_check"
    subprocess.run([gxx, "-O2", "-std=c++17", "-I", str(ROOT / "segmentctscans_b200" / "csrc"), "-I",
                    str(ROOT / "include"), str(ROOT / "tests" / "cpp" / "march_check.cpp"), "-o", str(exe)],
                   check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
