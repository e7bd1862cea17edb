"""Learned-DBP inference in chains of layers on the tensor cores
(ldbp_chain_kernel) at the sizes where its tiling can go wrong: fields shorter
than a tile (the circular filter wraps inside it), around one and two tiles,
filters of 1 to 255 taps (their halo decides how many layers a launch chains),
layer counts around the chain length, and tiles that run in FP32 (wide power
range).

Reference: the FP64 restatement of the model (oracle/ldbp_ref.py).  Tolerance:
a product of 22-bit pairs is off by at most 3 2^-22 = 7e-7 per layer and the
layers' errors add like a random walk or slower through near-unitary filters:
sqrt(13) x 7e-7 < 5e-6 for the longest chain here.
"""
import numpy as np
import pytest

import focss_gb300 as fg
from focss_gb300.ldbp import LearnedDBP
from oracle import ldbp_ref as R
from conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL = 5e-6


def model(rng, ctx, spans, steps, T, Tm, N, B, scale=0.95):
    L = spans * steps
    noise = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)  # noqa: E731
    # one dominant tap and a tail: near-unitary, so that errors do not grow
    h = noise(L, T) * 0.2 / np.sqrt(2 * T)
    h[:, T // 2] += 1.0
    xi = rng.standard_normal(L) * 0.1
    hmf = noise(Tm) / np.sqrt(2 * Tm)
    h, xi, hmf = h.astype(np.complex64), xi.astype(np.float32), hmf.astype(np.complex64)
    m = LearnedDBP(spans, steps, T, Tm, N, B, scale, ctx=ctx)
    m.set_params(h, xi, hmf)
    want = lambda x: R.forward(h.astype(complex), xi.astype(float), hmf.astype(complex), x.astype(complex),  # noqa: E731
                               float(np.float32(scale)), spans, steps)[..., 0::2]
    return m, want


def run(m, x, ctx):
    f = fg.Field(fg.Domain(1, x.shape[-1], 1.0), data=x[:, None, :], batch=x.shape[0], ctx=ctx)
    return m.forward(f).numpy()[:, 0]


@pytest.mark.parametrize("T,Tm", [(1, 1), (3, 15), (17, 33), (63, 255), (255, 63)])
@pytest.mark.parametrize("N", [40, 300, 1800, 2048, 2050, 4300])
def test_lengths_and_taps(ctx, T, Tm, N):
    rng = np.random.default_rng(T + N)
    m, want = model(rng, ctx, 2, 2, T, Tm, N, 2)
    x = ((rng.standard_normal((2, N)) + 1j * rng.standard_normal((2, N))) * 0.7).astype(np.complex64)
    assert rel_l2(run(m, x, ctx), want(x)) < TOL


@pytest.mark.parametrize("spans,steps", [(1, 1), (1, 5), (3, 3), (2, 4), (13, 1)])
def test_chain_lengths(ctx, spans, steps):
    rng = np.random.default_rng(spans * 10 + steps)
    m, want = model(rng, ctx, spans, steps, 63, 31, 3000, 1)
    x = ((rng.standard_normal((1, 3000)) + 1j * rng.standard_normal((1, 3000))) * 0.7).astype(np.complex64)
    assert rel_l2(run(m, x, ctx), want(x)) < TOL


def test_tiles_in_fp32(ctx):
    """A burst 60 dB above the rest of the field, and another field of a batch
    with a NaN: the finite field keeps its accuracy away from the burst too."""
    rng = np.random.default_rng(3)
    m, want = model(rng, ctx, 1, 3, 31, 15, 6000, 2)
    x = ((rng.standard_normal((2, 6000)) + 1j * rng.standard_normal((2, 6000))) * 1e-3).astype(np.complex64)
    x[0, 3000:3040] *= 1e3
    x[1, 100] = np.nan
    y, w = run(m, x, ctx), want(x)
    assert rel_l2(y[0], w[0]) < TOL
    assert rel_l2(y[0, :1400], w[0, :1400]) < TOL
    assert np.array_equal(np.isnan(y[1]), np.isnan(w[1]))


def test_parameters_can_change(ctx):
    """New parameters and an optimizer step reach the next pass."""
    rng = np.random.default_rng(4)
    m, want = model(rng, ctx, 1, 2, 15, 15, 512, 1)
    x = ((rng.standard_normal((1, 512)) + 1j * rng.standard_normal((1, 512))) * 0.7).astype(np.complex64)
    assert rel_l2(run(m, x, ctx), want(x)) < TOL
    t = fg.Field(fg.Domain(1, 256, 2.0), data=np.ones((1, 1, 256), np.complex64), ctx=ctx)
    m.loss_grad(fg.Field(fg.Domain(1, 512, 1.0), data=x[:, None], ctx=ctx), t)
    m.adam_step(1e-2)
    (h, xi, hmf), _ = m.get_params()
    now = R.forward(h, xi, hmf, x.astype(complex), float(np.float32(0.95)), 1, 2)[..., 0::2]
    assert rel_l2(run(m, x, ctx), now) < TOL
    assert rel_l2(now, want(x)) > 1e-3
