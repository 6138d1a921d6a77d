"""The tile shape and segment length that the library chooses by a volume's size give the bits of the
split form: volumes of one tile and of many, ragged slices and rows, every K and storage."""
import numpy as np
import pytest

from segmentctscans_b200 import potts
from tests._cases import TAU, random_volume

pytestmark = pytest.mark.gpu

# n, rows, cols, r: one slice; fewer items than multiprocessors; ragged last tiles; a few waves
SIZES = [(1, 20, 23, 8.7), (64, 33, 31, 14.2), (130, 90, 71, 33.4), (70, 150, 160, 70.6)]


@pytest.mark.parametrize("size", SIZES, ids=["-".join(map(str, s[:3])) for s in SIZES])
@pytest.mark.parametrize("K,storage,arith", [(2, "f32", "fast"), (3, "f32", "exact"), (3, "f32", "fast"),
                                             (3, "bf16", "fast"), (4, "f32", "exact"), (5, "f16", "fast"),
                                             (6, "f32", "fast")])
def test_chosen_tiling_equals_split(cuda_device, size, K, storage, arith):
    m, u, ci = random_volume(*size, K, seed=K + size[0])
    a = potts.solve(m, u, ci, 30.0, TAU, TAU, 8, variant=0, arith=arith, storage=storage)
    b = potts.solve(m, u, ci, 30.0, TAU, TAU, 8, variant=1, arith=arith, storage=storage)
    mv = m.mask_values
    for name in ("V", "Xi", "labels"):
        assert np.array_equal(mv(getattr(a, name)), mv(getattr(b, name))), name
    np.testing.assert_array_equal(a.stats.dq_trace, b.stats.dq_trace)


def test_context_rechooses_for_another_volume(cuda_device):
    """One context, volumes of different size in turn: the choice kept for a mapping is not used for another."""
    vols = [random_volume(*s, 3, seed=i) for i, s in enumerate(SIZES)]
    with potts.make_context(0) as ctx:
        for m, u, ci in vols + vols[::-1]:
            for arith in ("exact", "fast"):
                f = potts.solve_host(ctx, m, u, ci, 30.0, TAU, TAU, 6, arith=arith, stats=True)
                p = potts.solve_host(ctx, m, u, ci, 30.0, TAU, TAU, 6, arith=arith, stats=True, variant=1)
                np.testing.assert_array_equal(f.dq_trace, p.dq_trace)


def test_batch_runs_again_after_other_calls_of_its_context(cuda_device):
    """The captured graphs hold device addresses of the context: denoising and solves in between leave
    them valid."""
    import torch

    m, u, ci = random_volume(*SIZES[1], 3, seed=3)
    du, lab = torch.from_numpy(u).cuda(), torch.zeros(m.span, dtype=torch.uint8, device="cuda")
    g = du.clone()
    torch.cuda.synchronize()
    with potts.make_context(0) as ctx:
        with potts.Batch(ctx, [potts.BatchVolume(m, du.data_ptr(), ci, 30.0, labels_ptr=lab.data_ptr())], TAU, TAU,
                         9) as b:
            first = b.run().dq_trace.copy()
            potts.tv_denoise(ctx, m, g.data_ptr(), 0.06, 0.16, 3)
            potts.solve_host(ctx, m, u, ci, 30.0, TAU, TAU, 3, arith="fast")
            np.testing.assert_array_equal(b.run().dq_trace, first)
