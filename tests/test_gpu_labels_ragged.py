"""Label-finding inputs on lines whose slice count is not a multiple of four (16-byte loads with a partial
last quad) and on unaligned fields, and the 2-D histogram's cell selection
at its extremes (fewer cells than slots, all counts equal, one cell), against the oracle."""
import numpy as np
import pytest

from segmentctscans_b200 import potts
from tests._cases import random_volume

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 1], ids=["aligned", "unaligned"])
@pytest.mark.parametrize("n", [1, 3, 33, 130, 257, 319])
def test_ragged_lines(cuda_device, oracle_mod, n, shift):
    import torch

    m, u, _ = random_volume(n, 24, 31, 11.3, 3, seed=n)
    # values in the padding that would change every result
    u.reshape(m.n_lines, m.nstride)[:, n:] = 1e9
    buf = torch.zeros(m.span + 4, device="cuda")
    grad = torch.zeros(m.span + 4, device="cuda")
    buf[shift: shift + m.span] = torch.from_numpy(u).cuda()
    pu, pv = buf.data_ptr() + 4 * shift, grad.data_ptr() + 4 * shift
    with potts.make_context(0, stream=torch.cuda.current_stream().cuda_stream) as ctx:
        lo, hi = potts.min_max(ctx, m, pu)
        potts.grad_magn(ctx, m, pu, pv)
        counts, _, clo, chi = potts.calc_hist_auto(ctx, m, pu, 500)
        torch.cuda.synchronize()
        v = grad[shift: shift + m.span].cpu().numpy()
        assert (lo, hi) == (clo, chi) == oracle_mod.min_max(m, u)
        assert np.array_equal(m.mask_values(v), m.mask_values(oracle_mod.grad_magn(m, u)))
        assert np.array_equal(counts, oracle_mod.calc_hist(m, u, lo, hi, 500))
        for nb in (1, 60, 300):
            hist = potts.uv_hist(ctx, m, pu, pv, lo, hi, -1.0, 1.0, nb)
            assert np.array_equal(hist, oracle_mod.uv_hist(m, u, v, lo, hi, -1.0, 1.0, nb))


@pytest.mark.parametrize("nb", [7, 512, 1000])
def test_cell_selection(cuda_device, oracle_mod, nb):
    m, u, _ = random_volume(64, 40, 40, 19.1, 3, seed=nb)
    rng = np.random.default_rng(nb)
    flat = np.full_like(u, 0.5)
    spread = rng.random(u.size).astype(np.float32)
    with potts.make_context(0) as ctx:
        for a, b in ((u, spread), (flat, flat), (spread, rng.random(u.size).astype(np.float32))):
            fa, fb = potts.upload(ctx, m, a), potts.upload(ctx, m, b)
            hist, r = potts.uv_hist_auto(ctx, m, fa.data_ptr(), fb.data_ptr(), nb)
            assert np.array_equal(hist, oracle_mod.uv_hist(m, a, b, *r, nb))
            fa.free()
            fb.free()
