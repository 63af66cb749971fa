"""max_bfs_passes: a BFS that needs more passes ends the solve with
JFC_ERR_NOT_CONVERGED, and what it leaves (queued tiles, flagged regions, an ended
run of cycles) does not reach the next solve of the same graph, which is exact."""
import numpy as np
import pytest

import jfcut
import oracle
from conftest import zero_boundary

pytestmark = pytest.mark.gpu


def corridor(shape):
    """One corridor winding through the grid, more excess at its start than the deficit at its
    end takes: the relabel goes its whole way back, the cut its whole way on."""
    h, w = shape[-2:]
    open_ = np.zeros(shape, bool)
    cells = []
    for z in range(shape[0] if len(shape) == 3 else 1):
        rows = list(range(0, h, 2))
        plane = []
        for i, y in enumerate(rows):
            xs = range(w) if i % 2 == 0 else range(w - 1, -1, -1)
            plane += [(y, x) for x in xs]
            if y + 2 < h:
                plane.append((y + 1, plane[-1][1]))
        if z % 2:
            plane.reverse()
        cells += [((z,) + c if len(shape) == 3 else c) for c in plane]
    for c in cells:
        open_[c] = True
    caps = []
    axes = [(len(shape) - 1, 1), (len(shape) - 2, 1)] + ([(0, 1), (0, -1)] if len(shape) == 3 else [])
    axes += [(len(shape) - 2, -1), (len(shape) - 1, -1)]
    for axis, step in axes:
        caps.append(np.where(open_ & np.roll(open_, -step, axis), 50, 0).astype(np.int32).ravel())
    zero_boundary(shape, caps)
    e = np.zeros(shape, np.int32)
    e[cells[0]], e[cells[-1]] = 40, -10
    return e.ravel(), caps


@pytest.mark.parametrize("use_graph", [0, 1])
@pytest.mark.parametrize("shape", [(60, 210), (9, 20, 100)])
def test_budget_then_exact(ctx, shape, use_graph):
    e, caps = corridor(shape)
    flow, _, _, lab = oracle.maxflow(shape, e, caps)
    assert flow == 10 and lab.sum() > 1000
    g = jfcut.Graph(ctx, shape)
    for reload in (False, True):
        ctx.set_params(max_bfs_passes=1, use_graph=use_graph)
        g.set(e, caps)
        with pytest.raises(jfcut.JfcError) as ei:
            g.solve()
        assert ei.value.code == jfcut.ERR_NOT_CONVERGED
        ctx.reset_params()
        ctx.set_params(use_graph=use_graph)
        if reload:
            g.set(e, caps)
        assert g.solve().status == 0
        assert g.flow() == flow and np.array_equal(g.labels().ravel(), lab)
    g.close()
