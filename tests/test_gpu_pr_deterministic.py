"""A push-relabel visit reads its tile under one height vector, so a solve by parity
sweeps whose schedule does not follow the clock leaves the same residual state
every time: e, the arcs and the heights of repeated solves are equal, word by word."""
import numpy as np
import pytest

import jfcut
from conftest import zero_boundary

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,kw", [((70, 210), {}), ((515, 770), {}), ((515, 770), dict(tile_rows=16)),
                                      ((515, 770), dict(tile_rows=16, pr_mode=2)), ((13, 75, 130), {}),
                                      ((13, 75, 130), dict(tile_rows=16, tile_depth=4))])
def test_repeated_solves_leave_the_same_state(ctx, shape, kw):
    rng = np.random.default_rng(5 + len(shape))
    n = int(np.prod(shape))
    caps = [np.where(rng.random(n) < 0.8, rng.integers(1, 25, n), 0).astype(np.int32) for _ in range(2 * len(shape))]
    zero_boundary(shape, caps)
    e = rng.integers(-4, 4, n).astype(np.int32)
    e[rng.integers(0, n, n // 300)] -= 400
    e[rng.integers(0, n, n // 200)] += 300
    # sweeps only, and an interval that neither the clock nor the tail doubles
    ctx.set_params(pr_sched=1, relabel_interval=3, relabel_interval_max=3, **kw)
    g = jfcut.Graph(ctx, shape)
    first = None
    for _ in range(6):
        g.set(e, caps)
        g.solve()
        ex, arcs, h = g.state()
        state = [ex.ravel(), h.ravel()] + [a.ravel() for a in arcs]
        if first is None:
            first = [a.copy() for a in state]
        assert all(np.array_equal(a, b) for a, b in zip(first, state))
    g.close()
