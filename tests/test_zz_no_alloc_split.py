"""The allocation-free entry point uses the FFT split that focss_ssfm_run uses
for a length unless another one is pinned or autotuned: the same bits, at every
length it takes.  Collected with test_zz_no_alloc.py, after the other tests.
"""
import ctypes as C

import numpy as np
import pytest

import focss_gb300 as fg
from focss_gb300._lib import lib
from conftest import ALPHA, BETA2, GAMMA

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [fg.SSFM.UNIFORM, fg.SSFM.ADAPTIVE])
@pytest.mark.parametrize("lg", range(8, 18))
def test_same_bits(lg, grid):
    ctx = fg.Context()  # no pinned splits
    n, dt, batch = 1 << lg, 1 / 256e9, 2
    fiber, ssfm = fg.Fiber(ALPHA, BETA2, GAMMA, 5e3), fg.SSFM(fg.Fiber(ALPHA, BETA2, GAMMA, 5e3), 8)
    if grid != fg.SSFM.UNIFORM:
        ssfm.set_grid(grid)
        ssfm.set_maximum_phase_shift(0.005)
        ssfm.set_maximum_step_size(1000.0)
    rng = np.random.default_rng(lg)
    x = (rng.standard_normal((batch, 1, n)) + 1j * rng.standard_normal((batch, 1, n))) * 0.03
    want, buf = (fg.Field(fg.Domain(1, n, dt), data=x, batch=batch, ctx=ctx) for _ in range(2))
    ssfm.run(want, 1.0)
    ctx.sync()
    fb, op = fiber.c(), ssfm.opts()
    assert lib().focss_ssfm_run_noalloc(ctx.stream, buf.device_ptr(), n, batch, dt, C.byref(fb), C.byref(op), 1.0,
                                        None) == 0
    assert np.array_equal(buf.numpy(), want.numpy())
