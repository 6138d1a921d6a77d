"""The tiled TV kernel over several tiles and segments, and its two ways of dividing, against the FP32
oracle: ragged last tiles, the halo slice and row of a tile, segment starts, lambda and differences of g
inside and outside the range in which the quotients come from reciprocals."""
import numpy as np
import pytest

from segmentctscans_b200 import potts
from tests._cases import random_volume

pytestmark = pytest.mark.gpu

TAU_TV = 0.99 / 6.0


def assert_same(m, u, lam, iters, oracle_mod):
    out, st = potts.tv_denoise_host(m, u, lam, TAU_TV, iters)
    ref, dq = oracle_mod.tv(m, u, lam, TAU_TV, iters, "f32")
    assert np.array_equal(m.mask_values(out), m.mask_values(ref))
    np.testing.assert_array_equal(st.dq_trace, dq)


@pytest.mark.parametrize("n", [127, 128, 129, 131, 260, 387])
def test_tiles_along_n(cuda_device, oracle_mod, n):
    m, u, _ = random_volume(n, 41, 90, 19.6, 3, seed=n)
    assert_same(m, u, 0.06, 7, oracle_mod)


def test_segments_along_columns(cuda_device, oracle_mod):
    m, u, _ = random_volume(16, 20, 400, 9.4, 3, seed=1)  # a short circle in a long box: one run of columns
    assert_same(m, u, 0.06, 6, oracle_mod)
    m, u, _ = random_volume(24, 160, 170, 79.5, 3, seed=2)
    assert_same(m, u, 0.06, 6, oracle_mod)


@pytest.mark.parametrize("lam", [-0.3, 1e-7, 3e7])
def test_lambda_outside_the_reciprocal_range(cuda_device, oracle_mod, lam):
    m, u, _ = random_volume(40, 30, 30, 14.1, 3, seed=3)
    assert_same(m, u, lam, 4, oracle_mod)


def test_tiny_and_zero_differences(cuda_device, oracle_mod):
    m, u, _ = random_volume(140, 30, 30, 14.1, 3, seed=4)
    rng = np.random.default_rng(5)
    tiny = u * np.float32(2.0) ** rng.integers(-120, 0, u.size).astype(np.float32)
    flat = np.where(rng.random(u.size) < 0.8, np.float32(0.0), u)
    for g in (tiny.astype(np.float32), flat.astype(np.float32), np.zeros_like(u)):
        assert_same(m, g, 0.06, 5, oracle_mod)
