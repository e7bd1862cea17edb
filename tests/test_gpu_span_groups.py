"""Span loops of several UNIFORM fields of one length (one branch of the graph,
each pass over all their realizations): exactly what each field gives alone,
for uneven step counts and batches in any order, one and two modes, amplifier
noise of each field's own seed, next to fields that stay branches of their own,
and again on a replay."""
import numpy as np
import pytest

import focss_gb300 as fg
from conftest import ALPHA, BETA2, F0, GAMMA

pytestmark = pytest.mark.gpu
G, NF = 10 ** (0.2 * 80 / 10), 10 ** 0.5


def fields(ctx, shapes, seed):
    rng = np.random.default_rng(seed)
    out = []
    for modes, n, batch, dt in shapes:
        x = (rng.standard_normal((batch, modes, n)) + 1j * rng.standard_normal((batch, modes, n))) * 0.02
        out.append(fg.Field(fg.Domain(modes, n, dt, F0), data=x.astype(np.complex64), batch=batch, ctx=ctx))
    return out


@pytest.mark.parametrize("modes", [1, 2])
@pytest.mark.parametrize("direction", ["forward", "backward"])
def test_groups_equal_single_fields(ctx, modes, direction):
    fib = fg.Fiber(ALPHA, BETA2, GAMMA, 80e3, kappa=8 / 9 if modes == 2 else 1.0)
    shapes = [(modes, 4096, 1, 1 / 64e9), (modes, 1 << 15, 2, 1 / 64e9), (modes, 4096, 3, 1 / 64e9),
              (modes, 4096, 2, 1 / 80e9), (modes, 1 << 15, 1, 1 / 64e9), (modes, 4096, 1, 1 / 64e9)]
    ks = [3, 1, 1, 5, 4, 3]
    a = fields(ctx, shapes, 1)
    solvers = [fg.SSFM(fib, k) for k in ks]
    solvers[5].set_grid(fg.SSFM.ADAPTIVE)  # not part of a group
    solvers[5].set_maximum_phase_shift(0.02)
    solvers[5].set_maximum_step_size(20e3)
    amp = fg.Amplifier(G, NF, seed=5)
    where = dict(after=fg.Amplifier.AMPLIFY) if direction == "forward" else dict(
        before=fg.Amplifier.DROP_POWER, direction=fg.SSFM.BACKWARD)
    for run in range(2):  # the second replays the graph, with other noise
        amp.seed = 5 + 100 * run
        b = [f.copy() for f in a]
        steps = fg.span_loop(a, fib, solvers, 3, amplifier=amp, counter0=7, **where)
        for i, f in enumerate(b):
            one = fg.Amplifier(G, NF, seed=amp.seed + i)
            (s,) = fg.span_loop([f], fib, [solvers[i]], 3, amplifier=one, counter0=7, **where)
            np.testing.assert_array_equal(a[i].numpy(), f.numpy())
            np.testing.assert_array_equal(steps[i], s)
            if i < 5:
                np.testing.assert_array_equal(s, [3 * ks[i]] * shapes[i][2])
