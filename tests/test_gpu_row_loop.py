"""Row passes whose CTAs take several row blocks (1024-sample rows, more blocks
than run at once): block counts around the switch, a chunk that crosses from one
realization to the next, one that ends early (fewer steps), two modes, and the
plain transforms, against the same work in small launches of one block per CTA --
the same arithmetic, so equal to the bit."""
import numpy as np
import pytest

import focss_gb300 as fg
from focss_gb300 import dsp
from conftest import ALPHA, BETA2, F0, GAMMA

pytestmark = pytest.mark.gpu


def field(ctx, x):
    return fg.Field(fg.Domain(x.shape[1], x.shape[2], 1 / 512e9, F0), data=x, batch=x.shape[0], ctx=ctx)


def data(B, M, N):
    rng = np.random.default_rng(B)
    x = (rng.standard_normal((B, M, N)) + 1j * rng.standard_normal((B, M, N))) * 0.02
    x *= np.linspace(0.2, 1.5, B)[:, None, None]  # adaptive runs of different lengths
    return x.astype(np.complex64)


@pytest.mark.parametrize("B,M,N", [(19, 1, 1 << 19), (20, 1, 1 << 19), (10, 2, 1 << 19), (10, 1, 1 << 20)])
@pytest.mark.parametrize("grid", ["uniform", "adaptive"])
def test_batches_equal_single_realizations(ctx, B, M, N, grid):
    fib = fg.Fiber(ALPHA, BETA2, GAMMA, 2e3)
    s = fg.SSFM(fib, 2)
    if grid == "adaptive":
        s.set_grid(fg.SSFM.ADAPTIVE)
        s.set_maximum_phase_shift(0.01)
        s.set_maximum_step_size(1000.0)
    x = data(B, M, N)
    f = field(ctx, x)
    s.run(f)
    got = f.numpy()
    for b in range(B):
        one = field(ctx, x[b:b + 1])
        s.run(one)
        np.testing.assert_array_equal(got[b], one.numpy()[0])


def test_plain_transforms(ctx):
    x = data(20, 1, 1 << 19)
    got = dsp.wdm_select(field(ctx, x), 0, 100e9).numpy()
    low = dsp.decimate(field(ctx, x), 8).numpy()
    for b in (0, 7, 19):
        np.testing.assert_array_equal(got[b], dsp.wdm_select(field(ctx, x[b:b + 1]), 0, 100e9).numpy()[0])
        np.testing.assert_array_equal(low[b], dsp.decimate(field(ctx, x[b:b + 1]), 8).numpy()[0])
