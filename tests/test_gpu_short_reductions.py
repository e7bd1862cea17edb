"""Decisions, error counts, pair sums and the phase search at the sizes where
their launches change: realizations up to and just beyond what one cluster
decides on its own (kClusterSamples), fewer samples than threads, several modes
and realizations; angle grids on both sides of the five-step search's range.

Reference: the formulas in FP64 numpy.  Decisions, counts and angles are exact
(the samples keep 1e-4 from every decision boundary); the sums differ by the
order of at most 2^16 FP64 additions, 2^16 x 2^-53 < 1e-11 relative.
"""
import numpy as np
import pytest

import focss_gb300 as fg
from focss_gb300 import dsp

pytestmark = pytest.mark.gpu
LEVELS = np.array([-3, -1, 3, 1]) / np.sqrt(10.0)


def symbols(rng, B, M, N, noise=0.15):
    c = rng.integers(0, 16, (B, M, N))
    t = LEVELS[c & 3] + 1j * LEVELS[c >> 2]
    r = t + noise * (rng.standard_normal(t.shape) + 1j * rng.standard_normal(t.shape))
    return (0.7 * t).astype(np.complex64), (0.7 * r).astype(np.complex64)


def field(x, ctx):
    return fg.Field(fg.Domain(x.shape[1], x.shape[2], 1.0), data=x, batch=x.shape[0], ctx=ctx)


def codes_of(x, power):
    """Nearest codes with the realizations' total power, and whether safely so."""
    z = x.astype(complex) / np.sqrt(power / (x.shape[1] * x.shape[2]))[:, None, None]
    out, safe = 0, True
    for v, shift in ((z.real, 0), (z.imag, 2)):
        d = np.abs(v[..., None] - LEVELS)
        out = out | (np.argmin(d, -1) << shift)
        safe = safe & (np.abs(np.abs(v) - 2 / np.sqrt(10)) > 1e-4) & (np.abs(v) > 1e-4)
    return out, safe


@pytest.mark.parametrize("B,M,N", [(1, 1, 1), (3, 1, 31), (2, 2, 4000), (2, 1, 16384), (1, 2, 8192), (2, 1, 16385),
                                   (1, 2, 30001)])
def test_decisions_and_counts(ctx, B, M, N):
    rng = np.random.default_rng(N + B)
    t, r = symbols(rng, B, M, N)
    pt, pr = (np.sum(np.abs(v.astype(complex)) ** 2, (1, 2)) for v in (t, r))
    want, safe = codes_of(r, pr)
    got = dsp.hd_sequence_16qam(field(r, ctx))
    assert np.array_equal(got[safe], want[safe])
    level = np.sqrt(pr / (M * N))[:, None, None]
    hard = dsp.hard_decision_16qam(field(r, ctx)).numpy()
    assert np.allclose(hard[safe], ((LEVELS[want & 3] + 1j * LEVELS[want >> 2]) * level)[safe], rtol=1e-6, atol=0)
    (ct, st), (cr, sr) = codes_of(t, pt), codes_of(r, pt)
    unsafe = 4 * np.sum(~(st & sr), (1, 2))
    x = ct ^ cr
    bits = sum((x >> k) & 1 for k in range(4)).sum((1, 2))
    ber = dsp.bit_error_rate_16qam(field(t, ctx), field(r, ctx))
    assert np.all(np.abs(np.rint(ber * 4 * M * N) - bits) <= unsafe)


@pytest.mark.parametrize("B,M,N", [(1, 1, 1), (3, 2, 511), (2, 1, 513), (2, 1, 40000)])
def test_pair_sums(ctx, B, M, N):
    rng = np.random.default_rng(N)
    t, r = symbols(rng, B, M, N)
    a, b = t.astype(complex), r.astype(complex)
    power, diff = np.sum(np.abs(a) ** 2, (1, 2)), np.sum(np.abs(a - b) ** 2, (1, 2))
    for _ in range(2):  # the counters are back at zero
        q2 = dsp.q2_factor(field(t, ctx), field(r, ctx))
        assert np.allclose(q2, -10 * np.log10(diff / power), rtol=1e-11, atol=1e-10)
    s = dsp.ScalarEqualizer().estimate(field(t, ctx), field(r, ctx))
    want = np.sum(np.conj(b) * a, (1, 2)) / np.sum(np.abs(b) ** 2, (1, 2))
    assert np.allclose(s, want, rtol=1e-11, atol=1e-12)


@pytest.mark.parametrize("steps", [1, 2, 7, 8, 9, 720, 65536, 65537])
def test_phase_search(ctx, steps):
    rng = np.random.default_rng(steps)
    t, r = symbols(rng, 6, 1, 600)
    r = r * np.exp(1j * np.array([0.0, 0.5, 2.0, 3.1, -1.0, -3.1]))[:, None, None].astype(np.complex64)
    r[0] = 0  # no phase at all: the first step
    got = dsp.PhaseShiftEqualizer(steps).estimate(field(t, ctx), field(r, ctx))
    c = np.sum(np.conj(t.astype(complex)) * r.astype(complex), (1, 2))
    grid = 2 * np.pi * np.arange(steps) / steps
    v = (c[:, None] * np.exp(1j * grid)).real
    assert got[0] == 0
    index = np.rint(got * steps / (2 * np.pi)).astype(int)
    best = v.max(1)
    assert np.all(best - v[np.arange(6), index] <= 1e-13 * np.abs(c))
    assert np.allclose(got, 2 * np.pi * index / steps, rtol=1e-15, atol=0)
    for batch in (6, 70):  # by value and from a table
        x = np.resize(r, (batch, 1, 600))
        ang = np.linspace(-3, 3, batch)
        y = dsp.rotate(field(x, ctx), ang).numpy()
        assert np.allclose(y, x * np.exp(1j * ang)[:, None, None], rtol=1e-6, atol=1e-6)
