"""Learned-DBP training in chains of layers (ldbp_chain_kernel<true> and the
tap gradients of all layers at once) at the sizes where its tiling can go
wrong: fields shorter than a tile, around one and two tiles, filters of 1 to
255 taps, layer counts around the chain length, and tiles that run in FP32.

Reference: the FP64 restatement of the model (oracle/ldbp_ref.py).  Tolerance:
forward and backward together pass 2 x 13 layers at most, each off by at most
7e-7 (fir_tc.cuh's products) and a few FP32 roundings, adding like a random
walk: sqrt(26) x 1e-6 = 5e-6, twice that for gradients as products of both.
"""
import numpy as np
import pytest

import focss_gb300 as fg
from oracle import ldbp_ref as R
from conftest import rel_l2
from test_gpu_ldbp_chains import model

pytestmark = pytest.mark.gpu
TOL = 1e-5


def check(m, ctx, x, tx, scale, spans, steps):
    B, N = x.shape
    loss = m.loss_grad(fg.Field(fg.Domain(1, N, 1.0), data=x[:, None], batch=B, ctx=ctx),
                       fg.Field(fg.Domain(1, N // 2, 2.0), data=tx[:, None], batch=B, ctx=ctx))
    (h, xi, hmf), got = m.get_params()
    want_loss, *want = R.loss_grad(h.astype(complex), xi.astype(float), hmf.astype(complex), x.astype(complex),
                                   tx.astype(complex), float(np.float32(scale)), spans, steps)
    assert abs(loss - want_loss) < TOL * want_loss
    for g, w in zip(got, want):
        assert rel_l2(g, w) < TOL


def data(rng, B, N):
    noise = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)  # noqa: E731
    return noise(B, N) * np.float32(0.7), noise(B, N // 2)


@pytest.mark.parametrize("T,Tm", [(1, 1), (17, 33), (63, 255), (255, 63)])
@pytest.mark.parametrize("N", [40, 1800, 2048, 2050, 4300])
def test_lengths_and_taps(ctx, T, Tm, N):
    rng = np.random.default_rng(T + N)
    m, _ = model(rng, ctx, 2, 2, T, Tm, N, 2)
    check(m, ctx, *data(rng, 2, N), 0.95, 2, 2)


@pytest.mark.parametrize("spans,steps", [(1, 1), (1, 5), (3, 3), (2, 4), (13, 1)])
def test_chain_lengths(ctx, spans, steps):
    rng = np.random.default_rng(spans * 10 + steps)
    m, _ = model(rng, ctx, spans, steps, 63, 31, 3000, 1, 0.9)
    check(m, ctx, *data(rng, 1, 3000), 0.9, spans, steps)


def test_tiles_in_fp32(ctx):
    """A burst 60 dB above the rest of field and target: the gradient's tiles
    around it leave the tensor cores' range too."""
    rng = np.random.default_rng(3)
    m, _ = model(rng, ctx, 2, 3, 31, 15, 6000, 2)
    x, tx = data(rng, 2, 6000)
    x *= np.float32(1e-3)
    tx *= np.float32(1e-3)
    x[:, 3000:3040] *= np.float32(1e3)
    tx[:, 1500:1520] *= np.float32(1e3)
    check(m, ctx, x, tx, 0.95, 2, 3)
