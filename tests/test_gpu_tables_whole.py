"""Capacity tables around the number of runs from which they are kept entry by entry
(an eighth of the entries, at least 4,096), against the restatement."""
import numpy as np
import pytest

import jfcut
import oracle

pytestmark = pytest.mark.gpu


# (a t-link table of 65,537 entries has 8,188, 8,192 and 8,196 runs at 1777, 1778 and 1779)
@pytest.mark.parametrize("lambda_t", [1, 1777, 1778, 1779, 70000])
@pytest.mark.parametrize("lambda_n", [4095, 24500, 200000])
@pytest.mark.parametrize("shape", [(60, 90), (4, 20, 45)])
def test_both_sides_of_the_line(ctx, shape, lambda_n, lambda_t):
    rng = np.random.default_rng(lambda_n)
    img = rng.integers(0, 256, shape + (3,)).astype(np.uint8)
    seeds = np.zeros(shape, np.uint8)
    seeds[..., 5, 3:40] = 1
    seeds[..., -4, 20:44] = 2
    model = dict(lambda_n=lambda_n, z_weight_pct=50, lambda_t=lambda_t, k_fg=3, k_bg=4, seed_cap=1000000,
                 kmeans_iters=8)
    g = jfcut.Graph(ctx, shape)
    g.build_from_image(img, seeds, jfcut.PIX_RGB8, model)
    e_dev, r_dev, _ = g.state()
    e, caps, _ = oracle.build_graph(img, seeds, jfcut.PIX_RGB8, model)
    assert np.array_equal(e_dev.ravel(), e)
    assert all(np.array_equal(r.ravel(), c) for r, c in zip(r_dev, caps))
    g.close()
