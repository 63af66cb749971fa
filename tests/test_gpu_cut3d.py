"""The 3D cut and relabel on volumes whose sides fall on, just inside and just
outside the edges of a block of the cut (32 x 8 x 4 nodes, 32 x 16 x 2 for tiles
of 16 rows) for every tile shape: a percolating set of arcs carries reached nodes
through many blocks.  Heights are the exact residual BFS distances, flow and cut
are the oracle's (equal, no tolerance), also after a warm edit."""
import numpy as np
import pytest

import jfcut
import oracle
from conftest import zero_boundary

pytestmark = pytest.mark.gpu
SHAPES = [(1, 1, 1), (4, 8, 32), (5, 9, 33), (3, 7, 31), (2, 16, 32), (3, 17, 64), (9, 33, 97), (33, 5, 65), (1, 41, 100)]
TILES = [(8, 2), (8, 1), (16, 4), (16, 2), (16, 1)]


@pytest.mark.parametrize("rows,depth", TILES)
@pytest.mark.parametrize("shape", SHAPES)
def test_cut_at_block_edges(ctx, shape, rows, depth):
    rng = np.random.default_rng(shape[0] * 13 + shape[1] * 5 + shape[2])
    n = int(np.prod(shape))
    caps = [np.where(rng.random(n) < 0.4, rng.integers(1, 30, n), 0).astype(np.int32) for _ in range(6)]
    zero_boundary(shape, caps)
    e = np.zeros(n, np.int32)
    e[rng.integers(0, n, max(1, n // 2000))] = -50
    src = rng.integers(0, n, max(1, n // 500))
    e[src] += 90
    ctx.set_params(tile_rows=rows, tile_depth=depth)
    g = jfcut.Graph(ctx, shape)
    g.set(e, caps)
    sink = int(np.maximum(-e.astype(np.int64), 0).sum())
    for turn in range(2):
        g.solve()
        flow, _, _, lab = oracle.maxflow(shape, e, caps)
        er, r, h = g.state()
        d = oracle.sink_distances(shape, er, r)
        d[d == oracle.ORC_INF] = 1 << 30
        assert np.array_equal(h, d)
        assert np.array_equal(g.labels().ravel(), lab)
        # (the oracle solves the net excess; what cs and ct of one node cancel flows too)
        assert g.flow() == flow + sink - int(np.maximum(-e.astype(np.int64), 0).sum())
        idx = np.unique(np.concatenate([[0, n - 1], rng.integers(0, n, max(1, n // 300))])).astype(np.uint32)
        add = rng.integers(1, 60, idx.size).astype(np.int32)
        g.edit_tlinks(idx, add, np.zeros(idx.size, np.int32))
        e[idx] += add
    g.close()
