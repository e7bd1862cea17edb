"""Calls whose results are complete when they return: the stream of the context
is idle then, whatever was queued on it before."""
import numpy as np
import pytest

import focss_gb300 as fg
from focss_gb300 import dsp
from focss_gb300._lib import check, lib
from conftest import ALPHA, BETA2, GAMMA

pytestmark = pytest.mark.gpu

CALLS = {
    "wdm_mux": lambda f: dsp.wdm_mux(f, 1e9),
    "cd_compensation": lambda f: fg.cd_compensation(f, fg.Fiber(ALPHA, BETA2, GAMMA, 80e3), 2),
    "rotate": lambda f: dsp.rotate(f, 0.3),
    "scale_each": lambda f: dsp.scale_each(f, 0.5 - 0.2j),
}


@pytest.mark.parametrize("call", list(CALLS))
def test_stream_is_idle(ctx, call):
    torch = pytest.importorskip("torch")
    B, N = 3, 4096
    f = fg.Field(fg.Domain(1, N, 1 / 64e9), data=np.ones((B, 1, N), np.complex64), batch=B, ctx=ctx)
    big = fg.Field(fg.Domain(1, 1 << 20, 1 / 64e9), batch=16, ctx=ctx)
    check(lib().focss_bandpass(ctx.h, big.h, 1e9), ctx.h)
    CALLS[call](f)  # plans and kernels are in place
    ctx.sync()
    stream = torch.cuda.ExternalStream(ctx.stream)
    for _ in range(50):  # some milliseconds of work
        check(lib().focss_bandpass(ctx.h, big.h, 1e9), ctx.h)
    assert not stream.query()
    CALLS[call](f)
    assert stream.query()
