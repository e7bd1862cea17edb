"""A triplet sum that would be split over CTAs runs unsplit where there is no
memory for the partial sums.
"""
import ctypes as C

import numpy as np
import pytest

import focss_gb300 as fg
from focss_gb300 import sino
from focss_gb300._lib import lib
from conftest import rel_l2
from test_gpu_triplet_tiles import TOL, noise

pytestmark = pytest.mark.gpu


def test_without_room_for_partial_sums():
    """A sum whose groups would be split over CTAs (512 tiles), with no memory
    left for their partial sums (34 MB): it runs unsplit."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(12)
    m, n, _ = sino.diamond_terms(np.ones((41, 41)), 20)
    c = noise(rng, m.size)
    x = noise(rng, 1, 2, 2048 * 512)
    own = fg.Context()  # with no scratch yet
    f = fg.Field(fg.Domain(2, x.shape[2], 1 / 32e9), data=x, ctx=own)
    sino.triplet_apply(fg.Field(fg.Domain(2, 4100, 1 / 32e9), data=x[..., :4100], ctx=own), 20, m, n, c)
    out = fg.Field(f.domain, ctx=own)
    own.sync()
    mm, nn, cc = np.ascontiguousarray(m), np.ascontiguousarray(n), np.ascontiguousarray(c)
    held, size = [], 1 << 36
    try:
        while size >= 1 << 24:
            try:
                held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
            except torch.OutOfMemoryError:
                size //= 2
        status = lib().focss_triplet_apply(own.h, f.h, 20, mm.size, *(v.ctypes.data_as(C.c_void_p) for v in (mm, nn, cc)),
                                           out.h)
        own.sync()
    finally:
        held.clear()
        torch.cuda.empty_cache()
    assert status == 0
    assert rel_l2(out.numpy(), sino.triplet_apply(f, 20, m, n, c).numpy()) < TOL
