"""The 2D global relabel and cut on grids whose sides fall on, just inside and just
outside its region edges (64 rows x 6 words of 32 columns, 32 levels a phase)
and with distance caps around a phase's length: after a solve the heights are
the exact residual BFS distances, and flow and cut are the oracle's.  Sparse
deficits behind a percolating set of arcs make distances of several phases; a
warm edit then repeats both checks on changed arcs."""
import numpy as np
import pytest

import jfcut
import oracle
from conftest import zero_boundary

pytestmark = pytest.mark.gpu
SHAPES = [(1, 1), (16, 32), (64, 192), (65, 193), (63, 191), (128, 384), (129, 385), (33, 1100), (1100, 33), (97, 225)]


def check(g, shape, flow0):
    e, r, h = g.state()
    d = oracle.sink_distances(shape, e, r)
    d[d == oracle.ORC_INF] = 1 << 30
    assert np.array_equal(h, d)
    assert g.flow() == flow0


@pytest.mark.parametrize("rows", [8, 16])
@pytest.mark.parametrize("cap", [0, 1, 31, 32, 33, 97, -1])
@pytest.mark.parametrize("shape", SHAPES)
def test_heights_are_exact_at_region_edges(ctx, shape, cap, rows):
    rng = np.random.default_rng(shape[0] * 7 + shape[1] + 31 * max(cap, 0))
    n = shape[0] * shape[1]
    caps = [np.where(rng.random(n) < 0.62, rng.integers(1, 30, n), 0).astype(np.int32) for _ in range(4)]
    zero_boundary(shape, caps)
    e = np.zeros(n, np.int32)
    e[rng.integers(0, n, max(1, n // 4000))] = -200
    ctx.set_params(relabel_cap=cap, tile_rows=rows)
    g = jfcut.Graph(ctx, shape)
    g.set(e, caps)
    g.solve()
    check(g, shape, 0)
    # excess at a few nodes, among them the grid's corners
    idx = np.unique(np.concatenate([[0, n - 1, shape[1] - 1], rng.integers(0, n, max(1, n // 300))]))
    idx = idx[idx < n].astype(np.uint32)
    add = rng.integers(1, 60, idx.size).astype(np.int32)
    sink = -int(e.sum())   # sum of the sink capacities, which the edit leaves
    g.edit_tlinks(idx, add, np.zeros(idx.size, np.int32))
    e[idx] += add
    g.solve()
    flow, _, _, lab = oracle.maxflow(shape, e, caps)
    # (the oracle solves the net excess; what cs and ct of one node cancel flows too)
    check(g, shape, flow + sink - int(np.maximum(-e.astype(np.int64), 0).sum()))
    assert np.array_equal(g.labels().ravel(), lab)
    g.close()
