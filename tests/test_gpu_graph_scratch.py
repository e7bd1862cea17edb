"""Calls captured from the context's stream into a graph hold no scratch memory
that a later, larger call may replace, and leave no half-made tables behind:
replays and eager calls around them stay right.

References as in test_gpu_triplet_tiles.py and test_gpu_spectral_paths.py.
"""
import ctypes as C

import numpy as np
import pytest

import focss_gb300 as fg
from focss_gb300 import dsp, sino
from focss_gb300._lib import check, lib
from conftest import rel_l2
from test_gpu_ldbp_graphs import captured
from test_gpu_triplet_tiles import TOL, noise, reference

pytestmark = pytest.mark.gpu


def field(ctx, x):
    return fg.Field(fg.Domain(x.shape[1], x.shape[2], 1 / 32e9), data=x, batch=x.shape[0], ctx=ctx)


@pytest.mark.parametrize("first_seen", [True, False])
def test_triplet_sum(first_seen):
    ctx = fg.Context()
    rng = np.random.default_rng(2)
    m, n, _ = sino.diamond_terms(np.ones((25, 25)), 12)
    c = noise(rng, m.size)
    a, b = noise(rng, 1, 1, 5000), noise(rng, 1, 1, 5000)
    f, out = field(ctx, a), field(ctx, a)
    mm, nn, cc = np.ascontiguousarray(m), np.ascontiguousarray(n), np.ascontiguousarray(c)

    def call():
        check(lib().focss_triplet_apply(ctx.h, f.h, 12, mm.size, *(v.ctypes.data_as(C.c_void_p) for v in (mm, nn, cc)),
                                        out.h), ctx.h)
    if not first_seen:
        call()
    replay = captured(ctx, call)
    # an eager call with the same terms, before the graph ever ran, and a larger one
    assert rel_l2(sino.triplet_apply(f, 12, m, n, c).numpy(), reference(a, 12, m, n, c)) < TOL
    sino.triplet_apply(field(ctx, noise(rng, 1, 1, 1 << 18)), 12, m, n, c)
    f.upload(b)
    replay()
    assert rel_l2(out.numpy(), reference(b, 12, m, n, c)) < TOL


def test_pulse_shaping():
    ctx = fg.Context()
    rng = np.random.default_rng(3)
    s, t = noise(rng, 2, 1, 512), noise(rng, 2, 1, 512)
    f = field(ctx, s)
    want = dsp.rrc_shaping(field(ctx, t), 4, 0.1).numpy()
    out = dsp.rrc_shaping(f, 4, 0.1)
    replay = captured(ctx, lambda: check(lib().focss_rrc_shaping(ctx.h, f.h, 4, 0.1, 1.0, out.h), ctx.h))
    dsp.rrc_shaping(field(ctx, noise(rng, 4, 1, 1 << 16)), 4, 0.1)
    f.upload(t)
    replay()
    assert rel_l2(out.numpy(), want) < 1e-6
