"""Decimation whose row pass stores the kept bins itself (row_kernel_gather, launches
with enough rows) against the form that gathers them afterwards (a launch of one
realization): the same transform, so equal to the bit; and against FP64.  Every row
length, factors from none to the shortest output, odd and even splits, two modes.

Tolerance: FP32 transforms of up to 2^19 points, 19 x 6e-8 x 0.5 < 1e-6.
"""
import numpy as np
import pytest

import focss_gb300 as fg
from focss_gb300 import dsp
from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lg,rows,factors", [(9, 400, (1, 2)), (11, 160, (2, 8)), (13, 70, (1, 4, 32)), (15, 45, (8, 128)),
                                             (17, 12, (2, 16)), (18, 8, (4,)), (19, 6, (8, 2048))])
def test_rows_equal_single(ctx, lg, rows, factors):
    rng = np.random.default_rng(lg)
    N = 1 << lg
    x = (rng.standard_normal((rows // 2, 2, N)) + 1j * rng.standard_normal((rows // 2, 2, N))).astype(np.complex64)
    f = fg.Field(fg.Domain(2, N, 1.0), data=x, batch=rows // 2, ctx=ctx)
    for factor in factors:
        m = N // factor
        got = dsp.decimate(f, factor).numpy()
        for b in (0, rows // 2 - 1):
            one = dsp.decimate(fg.Field(fg.Domain(1, N, 1.0), data=x[b:b + 1, :1], ctx=ctx), factor).numpy()
            np.testing.assert_array_equal(got[b, 0], one[0, 0])
            s = np.fft.fft(x[b].astype(complex), axis=-1) / N
            want = np.fft.ifft(np.concatenate([s[..., :m // 2], s[..., N - m + m // 2:]], -1), axis=-1) * m
            assert rel_l2(got[b], want) < 1e-6
