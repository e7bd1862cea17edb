"""Learned-DBP calls captured from the context's stream into a graph: a replayed
forward pass uses the parameters of that moment, and a captured optimizer step
reaches the passes after its replay.

Reference and tolerance as in test_gpu_ldbp_chains.py.
"""
import numpy as np
import pytest

import focss_gb300 as fg
from focss_gb300._lib import check, lib
from focss_gb300.ldbp import LearnedDBP
from oracle import ldbp_ref as R
from conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL, N, T = 5e-6, 512, 15


def captured(ctx, call):
    torch = pytest.importorskip("torch")
    ctx.sync()
    s, g = torch.cuda.ExternalStream(ctx.stream), torch.cuda.CUDAGraph()
    with torch.cuda.stream(s):
        g.capture_begin(capture_error_mode="relaxed")
        call()
        g.capture_end()

    def replay():
        with torch.cuda.stream(s):
            g.replay()
        ctx.sync()
    return replay


class Case:
    def __init__(self, ctx):
        self.rng = np.random.default_rng(6)
        self.m = LearnedDBP(1, 2, T, T, N, 1, 0.95, ctx=ctx)
        self.x = self.noise(1, N) * np.float32(0.7)
        self.f = fg.Field(fg.Domain(1, N, 1.0), data=self.x[:, None], ctx=ctx)
        self.out = fg.Field(fg.Domain(1, N // 2, 2.0), ctx=ctx)
        self.ctx = ctx

    def noise(self, *s):
        return (self.rng.standard_normal(s) + 1j * self.rng.standard_normal(s)).astype(np.complex64)

    def new_params(self):
        h = self.noise(2, T) * np.float32(0.03)
        h[:, T // 2] += 1
        self.m.set_params(h, self.rng.standard_normal(2) * 0.1, self.noise(T) / np.float32(5))

    def forward(self):
        check(lib().focss_ldbp_forward(self.m.h, self.f.h, self.out.h), self.ctx.h)

    def right(self):
        h, xi, hmf = self.m.get_params()[0]
        want = R.forward(h, xi, hmf, self.x.astype(complex), float(np.float32(0.95)), 1, 2)[..., 0::2]
        return rel_l2(self.out.numpy()[:, 0], want) < TOL


def test_replayed_forward_uses_current_parameters(ctx):
    c = Case(ctx)
    c.new_params()
    c.forward()
    replay = captured(ctx, c.forward)
    for _ in range(2):
        c.new_params()
        replay()
        assert c.right()


def test_capture_leaves_the_next_call_right(ctx):
    c = Case(ctx)
    c.new_params()
    c.forward()
    c.new_params()
    captured(ctx, c.forward)  # recorded, not run
    c.forward()
    assert c.right()


def test_replayed_optimizer_step_reaches_the_next_pass(ctx):
    c = Case(ctx)
    c.new_params()
    c.m.loss_grad(c.f, fg.Field(fg.Domain(1, N // 2, 2.0), data=c.noise(1, 1, N // 2), ctx=ctx))
    replay = captured(ctx, lambda: c.m.adam_step(1e-2))
    c.forward()
    replay()
    c.forward()
    assert c.right()
