"""Transforms that read their input in place of a copy (channel selection,
decimation, matched filtering), pulse shaping from the repeated symbol spectrum
and dispersion compensation in one linear step: against FP64 numpy, at the
shortest and ordinary lengths, odd ratios of lengths' splits, several modes and
realizations, and with the input left as it was.

Tolerance: a forward and an inverse FP32 transform of up to 2^17 points, each
off by less than 17 x 6e-8 x 0.3, and one FP32 product: below 1e-6.
"""
import numpy as np
import pytest

import focss_gb300 as fg
from focss_gb300 import dsp
from conftest import ALPHA, BETA2, rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-6


def noise(rng, *shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)


def field(x, ctx, dt=1.0):
    return fg.Field(fg.Domain(x.shape[1], x.shape[2], dt), data=x, batch=x.shape[0], ctx=ctx)


@pytest.mark.parametrize("B,M,N", [(1, 1, 256), (3, 2, 2048), (2, 1, 1 << 17)])
@pytest.mark.parametrize("channel", [0, 1])
def test_channel_selection(ctx, B, M, N, channel):
    rng = np.random.default_rng(N)
    x, bw = noise(rng, B, M, N), 0.2
    f = field(x, ctx)
    got = dsp.wdm_select(f, channel, bw)
    cut = int(0.5 * bw * N) + 1
    s = np.fft.fft(x.astype(complex) * np.exp(-2j * np.pi * bw * channel * np.arange(N)), axis=-1)
    s[..., cut:N - cut + 1] = 0
    assert rel_l2(got.numpy(), np.fft.ifft(s, axis=-1)) < TOL
    assert np.array_equal(f.numpy(), x)


@pytest.mark.parametrize("N,factor", [(1024, 4), (1 << 16, 8)])
def test_decimation(ctx, N, factor):
    rng = np.random.default_rng(N)
    x, m = noise(rng, 2, 2, N), N // factor
    f = field(x, ctx)
    s = np.fft.fft(x.astype(complex), axis=-1) / N
    want = np.fft.ifft(np.concatenate([s[..., :m // 2], s[..., N - m + m // 2:]], -1), axis=-1) * m
    assert rel_l2(dsp.decimate(f, factor).numpy(), want) < TOL
    assert np.array_equal(f.numpy(), x)


@pytest.mark.parametrize("n,osf", [(128, 4), (256, 1), (256, 16), (2048, 2), (8192, 16)])
def test_shaping_and_matched_filter(ctx, n, osf):
    rng = np.random.default_rng(n + osf)
    x = noise(rng, 3, 2, n)
    f = field(x, ctx, float(osf))
    N = n * osf
    taps = np.fft.ifftshift(np.asarray(dsp.rrc_pulse(n, osf, 0.1)).astype(complex))
    up = np.zeros((3, 2, N), complex)
    up[..., ::osf] = x
    want = np.fft.ifft(np.fft.fft(up, axis=-1) * np.fft.fft(taps), axis=-1) / N * osf
    y = dsp.rrc_shaping(f, osf, 0.1)
    assert rel_l2(y.numpy(), want) < TOL
    y32 = y.numpy()
    back = np.fft.ifft(np.fft.fft(y32.astype(complex), axis=-1) * np.fft.fft(taps), axis=-1)[..., ::osf] / N
    assert rel_l2(dsp.rrc_sampling(y, osf, 0.1).numpy(), back) < TOL
    assert np.array_equal(y.numpy(), y32)


@pytest.mark.parametrize("B,M,N", [(2, 2, 256), (1, 1, 1 << 13), (3, 1, 1 << 16)])
def test_dispersion_compensation(ctx, B, M, N):
    rng = np.random.default_rng(N)
    dt, spans, length = 1 / 64e9, 20, 80e3
    x = noise(rng, B, M, N)
    f = field(x, ctx, dt)
    fg.cd_compensation(f, fg.Fiber(ALPHA, BETA2, 1.3e-3, length, 1.55e-6), spans)
    w = 2 * np.pi * np.fft.fftfreq(N, dt)
    want = np.fft.ifft(np.fft.fft(x.astype(complex), axis=-1) * np.exp(-0.5j * BETA2 * length * spans * w ** 2), axis=-1)
    assert rel_l2(f.numpy(), want) < TOL
