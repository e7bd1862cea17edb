"""Tiles of the tensor-core triplet sum that run in FP32 by several teams of
threads: as many as the terms' reach leaves room for (four, two and one), tiles of
which the field covers only a part, groups split over CTAs, one and two modes.

Reference as in test_gpu_triplet_tiles.py; every output is held to its tolerance
times the sum of the terms' magnitudes, so that the quiet ones count too.
"""
import numpy as np
import pytest

from test_gpu_triplet_tiles import TOL, apply, noise, reference

pytestmark = pytest.mark.gpu


def padded(a, radius, m, n, c):
    """reference() for offsets beyond the field's length."""
    pad = 7000
    y = reference(np.pad(a, [(0, 0), (0, 0), (pad, pad)]), 0, m, n, c)[..., pad:-pad]
    y[..., :radius] = y[..., a.shape[-1] - radius:] = 0
    return y


@pytest.mark.parametrize("reach", [20, 1500, 3000])
@pytest.mark.parametrize("modes", [1, 2])
@pytest.mark.parametrize("length", [900, 1500, 2048, 5000])
def test_wide_tiles(ctx, reach, modes, length):
    rng = np.random.default_rng(reach + length)
    a = noise(rng, 2, modes, length)
    a[..., 37::333] *= 300  # in every tile
    m = np.repeat(np.arange(-4, 5), 4)
    n = (np.array([0, 1, 3, 4]) + np.linspace(-reach, reach - 4, 9).astype(int)[:, None]).ravel()
    c = noise(rng, m.size)
    got, want = apply(ctx, a, 8, m, n, c), padded(a, 8, m, n, c)
    bound = abs(padded(np.abs(a), 8, m, n, np.abs(c)))
    assert np.all(np.abs(got - want) <= TOL * bound)
