"""The exact projection where a pair's |h|^2 leaves the range of the quotients from a reciprocal (2^40): the
IEEE operations, for one voxel of a pair and for both, give the FP32 oracle's bits in the fused (two voxels
per lane up to four labels, one above) and in the split form."""
import numpy as np
import pytest

from segmentctscans_b200 import potts
from tests._cases import TAU, random_volume

pytestmark = pytest.mark.gpu


# |q_i - q_j| is about tau2 times a difference of V: on both sides of 2^20, and beyond it
@pytest.mark.parametrize("tau2", [9e5, 4e6])
@pytest.mark.parametrize("K", [2, 3, 4, 5])
def test_long_corrections(cuda_device, oracle_mod, K, tau2):
    m, u, ci = random_volume(70, 24, 21, 9.8, K, seed=K)
    want = oracle_mod.solve(m, u, ci, 30.0, TAU, tau2, 3, precision="f32")
    mv = m.mask_values
    for variant in (0, 1):
        got = potts.solve(m, u, ci, 30.0, TAU, tau2, 3, variant=variant)
        for name in ("V", "Xi", "labels"):
            assert np.array_equal(mv(getattr(got, name)), mv(getattr(want, name))), (name, variant)
        np.testing.assert_array_equal(got.stats.dq_trace, want.dq_trace)
