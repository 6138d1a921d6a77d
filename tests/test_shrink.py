"""Dykstra's shrink without the square root's and divisions' branches (shrink_rn,
segmentctscans_b200/csrc/voxel.cuh), restated in C (tests/cpp/shrink_check.c), gives the IEEE results:
the root over every mantissa and every start value within the documented error of the GPU's reciprocal
square root, the quotients by the exceptional divisors over every numerator and by others at random."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_shrink_gives_the_ieee_results(tmp_path):
    gcc = shutil.which("gcc")
    if gcc is None:
        pytest.skip("no gcc")
    exe = tmp_path / "shrink_check"
    subprocess.run([gcc, "-O2", "-march=native", "-std=c11", "-ffp-contract=off", str(ROOT / "tests" / "cpp" / "shrink_check.c"), "-o",
                    str(exe), "-lm"], check=True, capture_output=True)
    r = subprocess.run([str(exe), "2000000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
