"""Learned-DBP chains whose samples leave the split's range inside a chain
(ldbp_chain_kernel checks every layer's input): the tile then runs in FP32, as a
tile does whose input is out of range, and an overflow stays within the reach of
the filters after it.

Reference: the FP64 restatement of the model (oracle/ldbp_ref.py).
"""
import numpy as np
import pytest

import focss_gb300 as fg
from focss_gb300.ldbp import LearnedDBP
from oracle import ldbp_ref as R
from conftest import rel_l2

pytestmark = pytest.mark.gpu


def taps(rng, L, T, gains):
    h = (rng.standard_normal((L, T)) + 1j * rng.standard_normal((L, T))) * 0.1 / np.sqrt(2 * T)
    h[:, T // 2] += 1.0
    return (h * np.asarray(gains)[:, None]).astype(np.complex64)


@pytest.mark.parametrize("layers,layer", [(3, 0), (3, 1), (6, 3)])
@pytest.mark.parametrize("at", [1000, 2040, 3000])
def test_overflow_in_a_middle_layer(ctx, layers, layer, at):
    """Sample `at` is 32 dB above the others and its power overflows at `layer`'s output
    (where the phase then is NaN); theirs do not.  Non-finite outputs: those whose
    filters read it, no others.  Tolerance of the others: that of FP32 filters,
    sqrt(layers x taps) roundings of 6e-8 of up to 1.5 times the sample, < 2e-6."""
    rng = np.random.default_rng(at + layer)
    T, N = 31, 4300
    x = ((rng.standard_normal((1, N)) + 1j * rng.standard_normal((1, N))) * 0.7).astype(np.complex64)
    x[0, at] = 38.0
    gains = np.ones(layers)
    gains[layer] = 1e18        # others: power 1e36 to 1e37
    gains[layer + 1] = 1e-18
    h = taps(rng, layers, T, gains)
    hmf = taps(rng, 1, T, [1.0])[0]
    m = LearnedDBP(1, layers, T, T, N, 1, 1.0, ctx=ctx)
    m.set_params(h, np.zeros(layers), hmf)
    y = m.forward(fg.Field(fg.Domain(1, N, 1.0), data=x[:, None], ctx=ctx)).numpy()[0, 0]
    want, acts = R.forward(h.astype(complex), np.zeros(layers), hmf.astype(complex), x.astype(complex), 1.0, 1, layers,
                           keep=True)
    bad = np.abs(acts[2 * layer + 1][0]) ** 2 > 3.4e38   # the layer's filter output
    assert bad[at] and np.sum(bad) < 4
    for _ in range(layers - layer):                      # the filters after it, the matched one among them
        bad = np.convolve(bad, np.ones(T), "same") > 0
    bad, want = bad[0::2], want[0, 0::2]
    assert not np.any(np.isfinite(y[bad]))
    assert np.all(np.isfinite(y[~bad]))
    assert rel_l2(y[~bad], want[~bad]) < 2e-6


@pytest.mark.parametrize("layer", [0, 2, 3])
@pytest.mark.parametrize("at", [700, 2045])
def test_gradient_range_grows_in_a_middle_layer(ctx, layer, at):
    """A sample whose phase at `layer` is xi p = 120: behind it the gradient
    there is some 46 dB above the rest.  Tolerance: that phase is off by up to
    2 x 120 x 1e-6 (twice the relative error of |y|), and so is each term of the
    gradients' sums; those of the gains cancel to 1/100 of their terms and less
    (plain complex64 evaluation of the model is off by 1e-3 there), so they are
    held against the sum of the terms' magnitudes."""
    rng = np.random.default_rng(at + layer)
    layers, T, N = 4, 31, 4300
    x = ((rng.standard_normal((1, N)) + 1j * rng.standard_normal((1, N))) * 0.05).astype(np.complex64)
    x[0, at] = 2.0
    h, hmf = taps(rng, layers, T, np.ones(layers)), taps(rng, 1, T, [1.0])[0]
    xi = np.full(layers, 0.01, np.float32)
    xi[layer] = 30.0
    tx = ((rng.standard_normal((1, N // 2)) + 1j * rng.standard_normal((1, N // 2))) * 0.05).astype(np.complex64)
    m = LearnedDBP(1, layers, T, T, N, 1, 1.0, ctx=ctx)
    m.set_params(h, xi, hmf)
    loss = m.loss_grad(fg.Field(fg.Domain(1, N, 1.0), data=x[:, None], ctx=ctx),
                       fg.Field(fg.Domain(1, N // 2, 2.0), data=tx[:, None], ctx=ctx))
    want_loss, *want = R.loss_grad(h.astype(complex), xi.astype(float), hmf.astype(complex), x.astype(complex),
                                   tx.astype(complex), 1.0, 1, layers)
    assert abs(loss - want_loss) < 2.4e-4 * want_loss
    gh, gxi, gmf = m.get_params()[1]
    assert rel_l2(gh, want[0]) < 2.4e-4
    assert rel_l2(gmf, want[2]) < 2.4e-4
    assert np.all(np.abs(gxi - want[1]) < 2.4e-4 * gain_terms(h.astype(complex), xi, hmf.astype(complex), x, tx, layers))


def gain_terms(h, xi, hmf, x, tx, layers):
    """sum |2 conj(g) p y| of each layer's gain gradient."""
    y, acts = R.forward(h, xi, hmf, x.astype(complex), 1.0, 1, layers, keep=True)
    g = np.zeros_like(y)
    g[..., 0::2] = (y[..., 0::2] - tx) / tx.size
    g = R.fir_adjoint(g, hmf)
    out = np.zeros(layers)
    for k in reversed(range(layers)):
        y = acts[2 * k + 1]
        p = np.abs(y) ** 2
        e = np.exp(1j * xi[k] * p)
        out[k] = np.sum(2 * np.abs(g) * p * np.abs(y))
        g = R.fir_adjoint(g * np.conj(e) * (1 - 1j * xi[k] * p) + np.conj(g) * 1j * xi[k] * y ** 2 * e, h[k])
    return out


@pytest.mark.parametrize("at", [900, 2044])
def test_one_overflowing_sample_in_silence(ctx, at):
    """Nothing else in the field: no run of samples to hold the overflow against."""
    rng = np.random.default_rng(at)
    layers, T, N = 3, 31, 4300
    x = np.zeros((1, N), np.complex64)
    x[0, at] = 38.0
    h = np.zeros((layers, T), np.complex64)
    h[:, T // 2] = [1e18, 1e-18, 1.0]
    hmf = taps(rng, 1, T, [1.0])[0]
    m = LearnedDBP(1, layers, T, T, N, 1, 1.0, ctx=ctx)
    m.set_params(h, np.zeros(layers), hmf)
    y = m.forward(fg.Field(fg.Domain(1, N, 1.0), data=x[:, None], ctx=ctx)).numpy()[0, 0]
    reach = np.abs(2 * np.arange(N // 2) - at) <= T // 2 * 3   # of two filters and the matched one
    assert not np.any(np.isfinite(y[reach]))
    assert not np.any(y[~reach])
