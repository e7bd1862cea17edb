"""Correction CNN at the sizes where a convolution's 128-position tiles and their
32-row stores end: sequences shorter than a warp's rows and than a tile, around one
and two tiles, and more tiles than CTAs.  Reference and tolerances as in
test_gpu_cnn.py (BF16 weights and activations)."""
import numpy as np
import pytest

import focss_gb300 as fg
from focss_gb300.cnn import CorrectionCNN, he_init
from oracle import cnn_ref as R
from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,L", [(3, 9), (2, 32), (2, 33), (1, 127), (2, 128), (2, 129), (1, 287), (3, 9000)])
def test_tile_edges(ctx, B, L):
    rng = np.random.default_rng(L)
    s = 0.3
    noise = lambda: rng.standard_normal((B, L)) + 1j * rng.standard_normal((B, L))  # noqa: E731
    y = (noise() * s).astype(np.complex64).astype(complex)
    tx = (y + 0.05 * noise()).astype(np.complex64).astype(complex)
    p = he_init(rng, zero_last=False) * 0.5
    net = CorrectionCNN(L, B, s, ctx=ctx)
    net.set_params(p)
    yf, tf = (fg.Field(fg.Domain(1, L, 1 / 32e9), data=v[:, None, :], batch=B, ctx=ctx) for v in (y, tx))
    z = net.forward(yf).numpy()[:, 0]
    loss = net.loss_grad(yf, tf)
    _, g = net.get_params()
    want_loss, want_g, want_z = R.loss_grad(p.astype(np.float64), y, tx, s)
    assert rel_l2(z, want_z) < 1e-3
    assert abs(loss - want_loss) < 1e-3 * want_loss
    off = 0
    for cin, cout in R.LAYERS:
        n = cout * R.KW * cin + cout
        assert rel_l2(g[off:off + n], want_g[off:off + n]) < 1e-2
        off += n
