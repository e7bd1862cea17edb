"""Fields that a call creates for its output are not cleared first: each such call
writes every sample, shown by handing it storage full of NaN (the context's pool
returns the block of a field just destroyed)."""
import numpy as np
import pytest

import focss_gb300 as fg
from focss_gb300 import dsp
from focss_gb300.cnn import CorrectionCNN
from focss_gb300.ldbp import LearnedDBP

pytestmark = pytest.mark.gpu
B, N = 3, 4096

CALLS = {
    "copy": lambda f: f.copy(),
    "map": lambda f: dsp.qam16_map(np.arange(B * N).reshape(B, 1, N) % 16, f.domain, batch=B, ctx=f.ctx),
    "upsample": lambda f: dsp.upsample(f, 2),
    "downsample": lambda f: dsp.downsample(f, 4),
    "decimate": lambda f: dsp.decimate(f, 4),
    "shaping": lambda f: dsp.rrc_shaping(f, 4, 0.1),
    "shaping_short": lambda f: dsp.rrc_shaping(dsp.downsample(f, 32), 4, 0.1),
    "sampling": lambda f: dsp.rrc_sampling(f, 2, 0.1),
    "select": lambda f: dsp.wdm_select(f, 1, 0.1),
    "select_centre": lambda f: dsp.wdm_select(f, 0, 0.1),
    "mux": lambda f: dsp.wdm_mux(f, 0.1),
    "hard": lambda f: dsp.hard_decision_16qam(f),
    "soft": lambda f: dsp.soft_decision_16qam(f, 0.1),
    "phase": lambda f: dsp.PhaseShiftEqualizer(16).train_equalize(f, f),
    "scalar": lambda f: dsp.ScalarEqualizer().train_equalize(f, f),
    "ldbp": lambda f: LearnedDBP(1, 2, 3, 5, N, B, 1.0, ctx=f.ctx).forward(f),
    "cnn": lambda f: CorrectionCNN(N, B, 1.0, ctx=f.ctx).forward(f),
}


@pytest.mark.parametrize("name", CALLS)
def test_every_sample_is_written(ctx, name):
    rng = np.random.default_rng(1)
    x = (rng.standard_normal((B, 1, N)) + 1j * rng.standard_normal((B, 1, N))).astype(np.complex64)
    f = fg.Field(fg.Domain(1, N, 1.0), data=x, batch=B, ctx=ctx)
    for n in (N // 32, N // 8, N // 4, N // 2, N, 2 * N, 4 * N):
        for b in (1, B):
            fg.Field(fg.Domain(1, n, 1.0), data=np.full((b, 1, n), np.nan, np.complex64), batch=b, ctx=ctx)
    assert np.all(np.isfinite(CALLS[name](f).numpy()))
