"""Triplet sums on the tensor cores (triplet_tc_kernel) at the sizes where its
tiling can go wrong: field lengths around the 1024- and 2048-output tiles and
the split of short fields over groups, dense runs around the 16-tap steps, shifted and one-sided runs, one and two modes, and the
tiles that take the FP32 sum instead (wide power range, non-finite samples).

Reference: the sum of src/focss/equalizer/sino.cpp:161-220 term by term in
complex128.  Tolerance: the FP16 pairs hold 22 bits of both factors and the
lo lo product (2^-22) is left out, so a product is off by at most 3 2^-22 =
7e-7; FP32 accumulation of T terms adds sqrt(T) 2^-24 < 1e-6 for T < 256.
"""
import numpy as np
import pytest

import focss_gb300 as fg
from focss_gb300 import sino
from conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL = 2e-6


def at(a, d):
    out = np.zeros_like(a)
    n = a.shape[-1]
    if d >= 0:
        out[..., :max(0, n - d)] = a[..., d:]
    else:
        out[..., -d:] = a[..., :n + d]
    return out


def reference(a, radius, m, n, c):
    a = a.astype(np.complex64).astype(np.complex128)
    c = np.asarray(c).astype(np.complex64).astype(np.complex128)
    y = np.zeros_like(a)
    with np.errstate(all="ignore"):
        for i in range(len(c)):
            t = np.sum(at(a, n[i]) * np.conj(at(a, m[i] + n[i])), axis=1, keepdims=True)
            y += c[i] * at(a, m[i]) * t
    k = np.arange(a.shape[-1])
    y[..., (k < radius) | (k >= a.shape[-1] - radius)] = 0
    return y


def noise(rng, *shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)) * 0.3


def apply(ctx, a, radius, m, n, c):
    f = fg.Field(fg.Domain(a.shape[1], a.shape[2], 1 / 32e9), data=a, batch=a.shape[0], ctx=ctx)
    return sino.triplet_apply(f, radius, m, n, c).numpy()


@pytest.mark.parametrize("modes", [1, 2])
@pytest.mark.parametrize("length", [257, 1023, 1024, 1025, 2047, 2048, 2049, 4100])
def test_tile_edges(ctx, modes, length):
    rng = np.random.default_rng(length)
    a = noise(rng, 2, modes, length)
    m, n, _ = sino.diamond_terms(np.ones((13, 13)), 6)
    c = noise(rng, m.size)
    assert rel_l2(apply(ctx, a, 6, m, n, c), reference(a, 6, m, n, c)) < TOL


# dense runs around the 1 / 17 / 33 tap limits of one, two and three steps, far
# from the centre on both sides, the longest run the path takes, and longer
@pytest.mark.parametrize("lo,hi", [(0, 0), (0, 1), (-4, 4), (-8, 8), (-8, 9), (-16, 16), (-16, 17), (40, 41), (-60, -57),
                                   (-104, 104), (-124, 124)])
@pytest.mark.parametrize("ms", [(0,), (-7, 3), (50, -50)])
def test_runs(ctx, lo, hi, ms):
    rng = np.random.default_rng(hi - lo)
    a = noise(rng, 1, 1, 1500)
    m, n = (v.ravel() for v in np.meshgrid(ms, np.arange(lo, hi + 1), indexing="ij"))
    c = noise(rng, m.size)
    assert rel_l2(apply(ctx, a, 3, m, n, c), reference(a, 3, m, n, c)) < TOL


@pytest.mark.parametrize("scale", [1e-9, 1.0, 1e9])
def test_scales_and_sparse_runs(ctx, scale):
    rng = np.random.default_rng(5)
    a = noise(rng, 1, 1, 1300) * scale
    m, n = np.array([0, 0, 2, 2, -9]), np.array([-30, 31, 4, 4, 0])  # holes and a repeated pair
    c = noise(rng, 5) / scale
    assert rel_l2(apply(ctx, a, 40, m, n, c), reference(a, 40, m, n, c)) < TOL


@pytest.mark.parametrize("bad", [np.nan, np.inf, 300.0])
def test_tiles_outside_the_split(ctx, bad):
    """One extreme sample: its tile takes the FP32 sum.  Outputs out of its
    reach keep their accuracy; a non-finite sample reaches every output that
    reads it and, through the zero taps that fill a run to whole groups of 8,
    at most 8 more."""
    rng = np.random.default_rng(8)
    a = noise(rng, 1, 1, 3000)
    a[0, 0, 1500] = bad
    m, n, _ = sino.diamond_terms(np.ones((11, 11)), 5)
    c = noise(rng, m.size)
    got, want = apply(ctx, a, 5, m, n, c)[0, 0], reference(a, 5, m, n, c)[0, 0]
    if np.isfinite(bad):
        assert rel_l2(got, want) < TOL
        far = np.abs(np.arange(3000) - 1500) > 5
    else:
        assert not np.any(np.isfinite(got[~np.isfinite(want)]))
        far = np.abs(np.arange(3000) - 1500) > 13
    assert rel_l2(got[far], want[far]) < TOL


def test_silent_field_and_term_cache(ctx):
    """Zeros give zeros, and term lists that share sizes are told apart."""
    m, n, _ = sino.diamond_terms(np.ones((9, 9)), 4)
    rng = np.random.default_rng(9)
    a = noise(rng, 1, 1, 1100)
    for _ in range(20):  # more lists than the cache keeps
        c = noise(rng, m.size)
        assert rel_l2(apply(ctx, a, 4, m, n, c), reference(a, 4, m, n, c)) < TOL
    assert not np.any(apply(ctx, np.zeros((1, 1, 1100), complex), 4, m, n, c))


@pytest.mark.parametrize("tiles", [100, 153, 400])
def test_splits_of_long_fields(ctx, tiles):
    """More tiles than SMs (and not), whose last wave splits fill: groups over
    several CTAs and their join, ragged end, against the reference."""
    rng = np.random.default_rng(tiles)
    a = noise(rng, 1, 1, 2048 * tiles - 1971)
    m, n, _ = sino.diamond_terms(np.ones((41, 41)), 20)
    keep = rng.permutation(m.size)[:60] if tiles > 200 else slice(None, None, 9)
    m, n = np.append(m[keep], np.arange(-20, 21)), np.append(n[keep], np.zeros(41, np.int32))
    c = noise(rng, m.size)
    assert rel_l2(apply(ctx, a, 40, m, n, c), reference(a, 40, m, n, c)) < TOL
