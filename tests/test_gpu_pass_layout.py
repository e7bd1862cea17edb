"""The two-pass layout with centred indices at every FFT length.

Rows and columns of the two passes stand for signed indices (col_work /
row_core in csrc/ssfm_kernels.cuh), which moves the wrap-around elements of
loads, stores, natural-order transposes, band-pass cuts and the decimation
gather.  Checked against numpy at every supported length, whose balanced
splits cover every sub-FFT length in both passes, and the Kerr rotation on
both sides of its small-phase bound (kKerrSmall).

Tolerances: an FP32 transform of 20 butterfly levels rounds each value by
2^-24 about twice a level, sqrt(40) 2^-24 = 3.8e-7 relative L2 per transform;
a Kerr phase of size phi is rounded to phi 2^-23 in FP32.
"""
import numpy as np
import pytest

import focss_gb300 as fg
from focss_gb300 import dsp
from conftest import F0, rel_l2

pytestmark = pytest.mark.gpu

LENGTHS = list(range(8, 21))


def _noise(rng, *shape):
    return ((rng.standard_normal(shape) + 1j * rng.standard_normal(shape)) * np.sqrt(0.5)).astype(np.complex64)


@pytest.mark.parametrize("lg", LENGTHS)
def test_natural_order_transforms(ctx, lg):
    n = 1 << lg
    x = _noise(np.random.default_rng(lg), 3, 1, n)
    f = fg.Field(fg.Domain(1, n, 1e-12, F0), data=x, batch=3, ctx=ctx)
    f.fft_inplace()
    assert rel_l2(f.numpy(), np.fft.fft(x.astype(np.complex128)) / n) < 1e-6
    f.ifft_inplace()
    assert rel_l2(f.numpy(), x) < 1e-6


@pytest.mark.parametrize("lg", LENGTHS)
@pytest.mark.parametrize("where", ["low", "half", "high"])
def test_bandpass_cut(ctx, lg, where):
    n = 1 << lg
    x = _noise(np.random.default_rng(100 + lg), 2, 1, n)
    f = fg.Field(fg.Domain(1, n, 1e-12, F0), data=x, batch=2, ctx=ctx)
    cut = {"low": 2, "half": n // 4 + 1, "high": n // 2 - 1}[where]
    y = dsp.bandpass_filter(f, (cut - 0.5) / (n * 1e-12))  # cut = int(frequency * duration) + 1
    s = np.fft.fft(x.astype(np.complex128))
    s[..., cut:n - cut + 1] = 0
    assert rel_l2(y.numpy(), np.fft.ifft(s)) < 2e-6


@pytest.mark.parametrize("lg", [10, 11, 13, 16, 19, 20])
@pytest.mark.parametrize("factor", [2, 4])
def test_decimate(ctx, lg, factor):
    n, m = 1 << lg, (1 << lg) // factor
    x = _noise(np.random.default_rng(200 + lg), 2, 1, n)
    f = fg.Field(fg.Domain(1, n, 1e-12, F0), data=x, batch=2, ctx=ctx)
    s = np.fft.fft(x.astype(np.complex128)) / n
    want = np.fft.ifft(np.concatenate([s[..., :m // 2], s[..., n - m // 2:]], -1)) * m
    assert rel_l2(dsp.decimate(f, factor).numpy(), want) < 2e-6


@pytest.mark.parametrize("lg", [8, 9, 11, 13, 15, 17, 18, 20])
@pytest.mark.parametrize("modes", [1, 2])
@pytest.mark.parametrize("phi", [0.02, 0.25, 6.0])
def test_kerr_phase_sizes(ctx, lg, modes, phi):
    """One Kerr-only step; the largest sample's phase is `phi` (6 rad: most
    threads take the general rotation; 0.25: on the bound)."""
    n = 1 << lg
    x = _noise(np.random.default_rng(300 + lg), 2, modes, n)
    p = np.sum(np.abs(x.astype(np.complex128)) ** 2, axis=1, keepdims=True)
    gamma = phi / p.max() / 1e3
    f = fg.Field(fg.Domain(modes, n, 1e-12, F0), data=x, batch=2, ctx=ctx)
    fg.SSFM(fg.Fiber(0.0, 0.0, gamma, 1e3), 1).run(f)
    want = x * np.exp(1j * gamma * 1e3 * p)
    assert rel_l2(f.numpy(), want) < 2e-6 + phi * 2.0 ** -23
