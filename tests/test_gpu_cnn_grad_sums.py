"""Weight and bias gradients of the correction CNN as sums over many positions,
each by itself: a network of single taps whose activations and gradients are known
exactly, so that the sums can be formed in 64 bits from the same BF16 factors.

Tolerance: a tensor-core accumulator that truncates after every 16 positions,
restated in float64, is off by up to 7e-7 over the 2048 positions a CTA sums; the
CTAs' sums add up in FP32 in any order, sqrt(300) roundings of 3e-8 relative to
their mean: below 3e-7.
"""
import numpy as np
import pytest

import focss_gb300 as fg
from focss_gb300.cnn import KW, CorrectionCNN, layout
from oracle.cnn_ref import bf16, shift

pytestmark = pytest.mark.gpu
TOL = 1e-6


def views(flat):
    return [(flat[w:w + int(np.prod(s))].reshape(s), flat[b:b + c]) for w, s, b, c in layout()[0]]


@pytest.mark.parametrize("mean", [1.0, 0.0])
@pytest.mark.parametrize("B,L", [(2, 4096), (12, 32768), (19, 32768)])
def test_sums_over_positions(ctx, B, L, mean):
    rng = np.random.default_rng(1)
    p = np.zeros(layout()[1], np.float32)
    (w1, _), (w2, _), (w3, _), (w4, _) = views(p)
    ch = np.arange(64)
    w1[ch, 4, ch % 2] = 0.5 ** (ch % 3)          # Re y or Im y, scaled
    w2[ch, 4, ch] = w3[ch, 4, ch] = 1
    w4[ch[:2, None] % 2, 4, ch.reshape(32, 2).T] = 2.0 ** -6
    y = ((rng.integers(1, 16, (B, L)) + 1j * rng.integers(1, 16, (B, L))) / 16).astype(np.complex64)
    noise = rng.standard_normal((B, L)) + 1j * rng.standard_normal((B, L))
    tx = (y - mean * (1 + 1j) + 0.5 * noise).astype(np.complex64)
    net = CorrectionCNN(L, B, 1.0, ctx=ctx)
    net.set_params(p)
    yf, tf = (fg.Field(fg.Domain(1, L, 1 / 32e9), data=v[:, None], batch=B, ctx=ctx) for v in (y, tx))
    d = net.forward(yf).numpy(np.complex64)[:, 0] - tx
    net.loss_grad(yf, tf)
    got = views(net.get_params()[1])

    x0, g4 = np.zeros((B, L, 16)), np.zeros((B, L, 16))
    inv = np.float32(1) / np.float32(B * L)
    for c, (a, b) in enumerate([(y.real, d.real), (y.imag, d.imag)]):
        x0[..., c], g4[..., c] = a, bf16((np.float32(2) * b) * inv)
    act = bf16(x0 @ w1[:, 4].T.astype(float))    # positive: ReLU passes it through the layers
    g = bf16(g4 @ w4[:, 4].astype(float))
    for (gw, gb), grad, inp in zip(got, (g, g, g, g4), (x0, act, act, act)):
        flat = grad.reshape(-1, grad.shape[-1])
        ww = np.stack([flat.T @ shift(inp, k - 4).reshape(-1, inp.shape[-1]) for k in range(KW)], 1)
        wb = flat.sum(0)
        assert np.linalg.norm(gw - ww) < TOL * np.linalg.norm(ww)
        assert np.linalg.norm(gb - wb) < TOL * np.linalg.norm(wb)
