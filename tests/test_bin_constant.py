"""The histogram kernels' bin by an added constant (hist_bin_r, segmentctscans_b200/csrc/kernels_hist.cuh)
restated in C (tests/cpp/bin_constant_check.c) gives the reference's bin for every value tested, as in
test_bin_rounding.py: random values, both ends of each range and every rounding boundary."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_bin_by_constant_matches_the_division(tmp_path):
    gcc = shutil.which("gcc")
    if gcc is None:
        pytest.skip("no gcc")
    exe = tmp_path / "bin_constant_check"
    subprocess.run([gcc, "-O2", "-std=c11", "-ffp-contract=off", str(ROOT / "tests" / "cpp" / "bin_constant_check.c"),
                    "-o", str(exe), "-lm"], check=True, capture_output=True)
    r = subprocess.run([str(exe), "500000"], capture_output=True, text=True, timeout=300)
    lines = [ln.split() for ln in r.stdout.splitlines() if ln.strip()]
    assert r.returncode == 0 and len(lines) == 11, r.stdout + r.stderr
    for start, end, nb, values, fallbacks, mismatches in lines:
        assert int(mismatches) == 0, (start, end, nb)
        assert int(values) > 500000
