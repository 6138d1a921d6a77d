"""Fields of noise, where nearly every voxel runs the projection loop in every plane and the row warps find
their queues full: the fused form gives the split form's bits, and the exact one the oracle's."""
import numpy as np
import pytest

from segmentctscans_b200 import potts
from segmentctscans_b200.layout import CylinderMapping
from tests._cases import TAU

pytestmark = pytest.mark.gpu


def noise(K, seed):
    m = CylinderMapping.cylinder(150, 61, 58, 28.4)
    rng = np.random.default_rng(seed)
    return m, rng.random(m.span, dtype=np.float32), [float(np.float32((i + 0.5) / K)) for i in range(K)]


@pytest.mark.parametrize("storage", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("arith", ["fast", "exact"])
@pytest.mark.parametrize("K", [2, 3, 4, 6])
def test_full_queues(cuda_device, oracle_mod, K, arith, storage):
    m, u, ci = noise(K, K)
    mv = m.mask_values
    ref = potts.solve(m, u, ci, 30.0, TAU, TAU, 12, variant=1, arith=arith, storage=storage)
    shapes = [{}, {"tile_rows": 8, "tile_slices": 128}] if K <= 3 else [{}]  # the second: named for K = 2 and 3
    for shape in shapes:
        got = potts.solve(m, u, ci, 30.0, TAU, TAU, 12, variant=0, arith=arith, storage=storage, **shape)
        for name in ("V", "Xi", "labels"):
            assert np.array_equal(mv(getattr(got, name)), mv(getattr(ref, name))), (name, shape)
        np.testing.assert_array_equal(got.stats.dq_trace, ref.stats.dq_trace)
    if storage == "f32" and arith == "exact" and K <= 4:
        want = oracle_mod.solve(m, u, ci, 30.0, TAU, TAU, 12, precision="f32")
        assert np.array_equal(mv(ref.V), mv(want.V))
