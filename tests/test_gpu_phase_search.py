"""The phase-shift equalizer's search where an FP32 argument does not do (more than
65536 steps) and where it tries all steps (fewer than 8, more than 2^24, or sums without
an argument): against numpy on the same grid.

Tolerance: the same step, as the FP64 sums are off by less than the difference
between neighbouring steps.
"""
import numpy as np
import pytest

import focss_gb300 as fg
from focss_gb300 import dsp

pytestmark = pytest.mark.gpu


def field(ctx, x):
    return fg.Field(fg.Domain(1, x.shape[-1], 1 / 32e9), data=x[:, None], batch=len(x), ctx=ctx)


@pytest.mark.parametrize("steps", [1, 3, 7, 65537, 100003, (1 << 24) - 1, (1 << 24) + 1])
def test_all_steps(ctx, steps):
    rng = np.random.default_rng(steps)
    d = (rng.standard_normal((4, 3000)) + 1j * rng.standard_normal((4, 3000))).astype(np.complex64)
    r = (d * np.exp(1j * np.array([0.0, 1.234, -3.1, 2.0]))[:, None]).astype(np.complex64)
    got = dsp.PhaseShiftEqualizer(steps).estimate(field(ctx, d), field(ctx, r))
    c = np.sum(np.conj(d.astype(complex)) * r, axis=1)
    # the steps around each peak (all of them when there are few)
    near = [np.arange(steps) if steps < 9 else int(round(-np.angle(v) / (2 * np.pi) * steps)) + np.arange(-4, 5) for v in c]
    want = [k[np.argmax((v * np.exp(2j * np.pi * k / steps)).real)] % steps * (2 * np.pi / steps) for k, v in zip(near, c)]
    assert np.allclose(got, want, rtol=0, atol=1e-9)


@pytest.mark.parametrize("value", [0.0, np.nan])
def test_no_argument(ctx, value):
    d = np.full((2, 500), value, np.complex64)
    assert not np.any(dsp.PhaseShiftEqualizer(720).estimate(field(ctx, d), field(ctx, d)))
