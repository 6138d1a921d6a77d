"""Tapes that take over an earlier tape's device buffers: the same results as tapes with buffers of their
own, in any order of sizes and lifetimes; the memory counts as available and comes back."""
import numpy as np
import pytest

from segmentctscans_b200 import potts
from tests._cases import TAU, random_volume

pytestmark = pytest.mark.gpu


def pass_through(ctx, vol, every):
    import torch

    m, u, ci, truth = vol
    du, dt = torch.from_numpy(u).cuda(), torch.from_numpy(truth).cuda()
    g = torch.zeros(m.span, device="cuda")
    torch.cuda.synchronize()
    with potts.Tape(ctx, m, du.data_ptr(), dt.data_ptr(), ci, 30.0, TAU, TAU, 9, every) as t:
        gc, gl = t.backward(g.data_ptr())
        loss = t.loss
    ctx.synchronize()
    return loss, g.cpu().numpy(), gc, gl


def volume(n, side, k, seed):
    m, u, ci = random_volume(n, side, side, 0.45 * side, k, seed=seed)
    rng = np.random.default_rng(seed)
    return m, u, ci, rng.integers(0, k, m.span).astype(np.uint8)


def test_reused_buffers_give_the_same_results(cuda_device):
    vols = [volume(24, 22, 3, 1), volume(24, 22, 3, 2), volume(40, 30, 3, 3), volume(24, 22, 4, 4), volume(9, 12, 2, 5)]
    alone = []
    for v in vols:
        with potts.make_context(0) as ctx:
            alone.append(pass_through(ctx, v, 4))
    with potts.make_context(0) as ctx:
        for i in (0, 1, 0, 2, 1, 3, 0, 4, 2):
            got = pass_through(ctx, vols[i], 4)
            assert got[0] == pytest.approx(alone[i][0], rel=1e-12)
            assert np.array_equal(got[1], alone[i][1])
            np.testing.assert_allclose(got[2], alone[i][2], rtol=1e-9, atol=1e-15)
            assert got[3] == pytest.approx(alone[i][3], rel=1e-9)


def test_two_tapes_at_once_and_a_tape_that_outlives_its_context(cuda_device):
    import torch

    m, u, ci, truth = volume(24, 22, 3, 1)
    du, dt = torch.from_numpy(u).cuda(), torch.from_numpy(truth).cuda()
    torch.cuda.synchronize()
    ctx = potts.make_context(0)
    args = (m, du.data_ptr(), dt.data_ptr(), ci, 30.0, TAU, TAU, 6, 3)
    a, b = potts.Tape(ctx, *args), potts.Tape(ctx, *args)
    g = [torch.zeros(m.span, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    b.backward(g[1].data_ptr())
    a.close()
    c = potts.Tape(ctx, *args)
    c.backward(g[0].data_ptr())
    ctx.synchronize()
    assert torch.equal(g[0], g[1])
    c.close()
    ctx.close()
    b.close()


def test_kept_memory_is_available_and_comes_back(cuda_device):
    v = volume(160, 150, 3, 6)
    with potts.make_context(0) as ctx:
        m, u, ci, _ = v
        potts.solve_host(ctx, m, u, ci, 30.0, TAU, TAU, 2)
        before = ctx.device_memory()[0]
        pass_through(ctx, v, 9)
        assert abs(ctx.device_memory()[0] - before) < 64 << 20
        import torch

        torch.cuda.empty_cache()
        kept = torch.cuda.mem_get_info()[0]
        potts.solve_host(ctx, m, u, ci, 30.0, TAU, TAU, 2)
        assert torch.cuda.mem_get_info()[0] > kept + (256 << 20)
