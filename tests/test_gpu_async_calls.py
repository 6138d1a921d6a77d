"""Calls that follow an asynchronous solve on its context and mapping, while its kernels still run: the work
items of another tile shape must not reach the solve (contexts with a stream of their own)."""
import numpy as np
import pytest

from segmentctscans_b200 import potts
from tests._cases import TAU, random_volume

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("follow", ["tv", "grad_magn", "other_labels", "other_arith"])
def test_work_items_of_the_next_call_stay_behind(cuda_device, follow):
    import torch

    m, u, ci = random_volume(96, 200, 190, 90.3, 3, seed=4)
    ci2 = [0.2, 0.8]
    du = torch.from_numpy(u).cuda()
    g, v = du.clone(), torch.zeros_like(du)
    lab = torch.zeros(m.span, dtype=torch.uint8, device="cuda")
    lab2 = torch.zeros_like(lab)
    torch.cuda.synchronize()
    with potts.make_context(0) as ctx:
        def solve(out, labels=ci, arith="fast", iters=150):
            potts.solve_device(ctx, m, du.data_ptr(), labels, 30.0, TAU, TAU, iters, labels_ptr=out.data_ptr(),
                               arith=arith, stats=False)

        def next_call():
            if follow == "tv":
                potts.tv_denoise(ctx, m, g.data_ptr(), 0.06, 0.16, 2, stats=False)
            elif follow == "grad_magn":
                potts.grad_magn(ctx, m, du.data_ptr(), v.data_ptr())
            elif follow == "other_labels":
                solve(lab2, labels=ci2, iters=3)
            else:
                solve(lab2, arith="exact", iters=3)

        solve(lab)
        ctx.synchronize()
        want = lab.clone()
        for _ in range(3):  # later passes find every buffer at its size: nothing waits
            lab.zero_()
            torch.cuda.synchronize()
            solve(lab)
            next_call()
            ctx.synchronize()
            assert torch.equal(lab, want)
        assert np.array_equal(m.mask_values(want.cpu().numpy()),
                              m.mask_values(potts.solve(m, u, ci, 30.0, TAU, TAU, 150, arith="fast").labels))
