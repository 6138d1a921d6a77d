"""TV denoising of fields that hold NaN and infinities: every form (tiled, split, per voxel) gives the
FP32 oracle's values, NaN where it has NaN.  A voxel with one NaN difference has a NaN |G|, which makes
all three of its dual components NaN."""
import numpy as np
import pytest

from segmentctscans_b200 import potts
from tests._cases import random_volume

pytestmark = pytest.mark.gpu

TAU_TV = 0.99 / 6.0


def field(m, u, kind, seed):
    """u with some in-mask voxels that are not finite."""
    rng = np.random.default_rng(seed)
    g = u.reshape(m.n_lines, m.nstride).copy()
    lines = rng.choice(m.n_lines, 6, replace=False)
    slices = rng.integers(0, m.n_images, 6)
    if kind == "one_nan":
        g[lines[0], slices[0]] = np.nan
    elif kind == "nans":
        g[lines, slices] = np.nan
    elif kind == "nan_run":  # whole quads of slices, and their edges
        g[lines[0], 1:min(11, m.n_images)] = np.nan
    elif kind == "infs":
        g[lines[:3], slices[:3]] = np.inf
        g[lines[3:], slices[3:]] = -np.inf
    else:  # mixed, with a finite value whose square overflows
        g[lines[0], slices[0]] = np.nan
        g[lines[1], slices[1]] = np.inf
        g[lines[2], slices[2]] = 3e38
    return g.reshape(-1)


@pytest.mark.parametrize("variant", [0, 1, 2], ids=["tiled", "plain", "fused_voxel"])
@pytest.mark.parametrize("kind", ["one_nan", "nans", "nan_run", "infs", "mixed"])
@pytest.mark.parametrize("n", [20, 133])
def test_non_finite_values(cuda_device, oracle_mod, n, kind, variant):
    m, u, _ = random_volume(n, 24, 23, 10.7, 3, seed=n)
    g = field(m, u, kind, seed=n + 1)
    for iters in (1, 4):
        out, _ = potts.tv_denoise_host(m, g, 0.06, TAU_TV, iters, variant=variant)
        ref, _ = oracle_mod.tv(m, g, 0.06, TAU_TV, iters, "f32")
        a, b = m.mask_values(out), m.mask_values(ref)
        assert np.isnan(b).any() and not np.isnan(b).all()
        np.testing.assert_array_equal(a, b)  # NaN equals NaN here
