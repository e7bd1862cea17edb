"""Tap gradients of learned filters longer than 97 taps (tap_grad_kernel gives
them several CTAs a tile, each with a window 128 samples further on) on fields
whose power steps by 40 dB near a window's edge: of one tile, some CTAs then sum
in FP32 and others on the tensor cores, and their shares have to add up.

Reference: the FP64 restatement of the model (oracle/ldbp_ref.py), filter by
filter and at each tap.  Tolerance as in test_gpu_ldbp_chain_grads.py.
"""
import numpy as np
import pytest

import focss_gb300 as fg
from oracle import ldbp_ref as R
from conftest import rel_l2
from test_gpu_ldbp_chains import model

pytestmark = pytest.mark.gpu
TOL = 1e-5
N, QUIET = 8192, np.float32(1e-2)


@pytest.mark.parametrize("loud_target", [False, True])
@pytest.mark.parametrize("rising", [False, True])
@pytest.mark.parametrize("offset", [-130, -97, -31, 0, 64, 127])
@pytest.mark.parametrize("T,Tm", [(99, 63), (63, 255), (255, 255)])
def test_power_step(ctx, T, Tm, offset, rising, loud_target):
    """The step lies `offset` samples from a multiple of the tile's 2048, and as
    the field is circular another one at sample 0; loud_target makes the target,
    and with it the gradient, loud where the field is quiet, so that the quiet
    tiles count as much as the others."""
    rng = np.random.default_rng(T + Tm + offset)
    noise = lambda n: (rng.standard_normal((1, n)) + 1j * rng.standard_normal((1, n))).astype(np.complex64)  # noqa: E731
    m, _ = model(rng, ctx, 1, 2, T, Tm, N, 1)
    x, tx = noise(N) * np.float32(0.7), noise(N // 2)
    quiet = slice(0, 4096 + offset) if rising else slice(4096 + offset, N)
    x[:, quiet] *= QUIET
    if loud_target:
        tx[:, slice(0, 2048) if rising else slice(2048, None)] /= QUIET
    loss = m.loss_grad(fg.Field(fg.Domain(1, N, 1.0), data=x[:, None], ctx=ctx),
                       fg.Field(fg.Domain(1, N // 2, 2.0), data=tx[:, None], ctx=ctx))
    (h, xi, hmf), (gh, _, gmf) = m.get_params()
    want_loss, wh, _, wmf = R.loss_grad(h.astype(complex), xi.astype(float), hmf.astype(complex), x.astype(complex),
                                        tx.astype(complex), float(np.float32(0.95)), 1, 2)
    assert abs(loss - want_loss) < TOL * want_loss
    for got, want in [(gh[0], wh[0]), (gh[1], wh[1]), (gmf, wmf)]:
        assert rel_l2(got, want) < TOL
        assert np.max(np.abs(got - want)) < TOL * np.linalg.norm(want)
