"""Triplet sums whose coefficients differ by orders of magnitude: a weak term
keeps its accuracy where the strong ones have no part in a symbol.

Reference and tolerance as in test_gpu_triplet_tiles.py.
"""
import numpy as np
import pytest

from conftest import rel_l2
from test_gpu_triplet_tiles import TOL, apply, noise, reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("same_run", [True, False])
@pytest.mark.parametrize("weak", [1e-3, 1e-6, 2.0 ** -28, 1e-9, 1e-12])
def test_weak_terms(ctx, weak, same_run):
    """The strong term (m = 0 or 3, n = 7) needs samples 7 apart, the weak ones
    samples 1 to 3 apart: pulses of four samples every 32 have only those."""
    rng = np.random.default_rng(11)
    a = noise(rng, 1, 1, 4100)
    a[..., np.arange(4100) % 32 >= 4] = 0
    m = np.array([0, 0, 0, 1, 1, 0 if same_run else 3])
    n = np.array([1, 2, 3, -1, 1, 7])
    c = noise(rng, m.size) * weak
    c[-1] = 0.9 - 0.4j
    got, want = apply(ctx, a, 8, m, n, c), reference(a, 8, m, n, c)
    assert rel_l2(got, reference(a, 8, m[:-1], n[:-1], c[:-1])) < TOL  # the strong term has no part
    assert rel_l2(got, want) < TOL
