"""What the threads of a block agree on (segmentctscans_b200/csrc/block.cuh), run on the host with the
threads as coroutines in unfavourable orders (tests/cpp/block_check.cpp): the list of loop voxels runs
every voxel once, with its own values, and its barriers pair up; when a wait gives up, all threads leave
their loop together."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_block_agrees_in_every_order(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    exe = tmp_path / "block_check"
    subprocess.run([gxx, "-O1", "-std=c++17", "-Wall", "-Werror", "-I", str(ROOT / "segmentctscans_b200" / "csrc"),
                    str(ROOT / "tests" / "cpp" / "block_check.cpp"), "-o", str(exe)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
