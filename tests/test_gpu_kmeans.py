"""Colour models (k-means over the seeds) against the CPU restatement, bit for
bit, through the t-links they give: seed lists around the block and cluster
sizes of the device kernel (1,024 seeds a block, 8 blocks a cluster, 131,072
seeds where it goes grid-wide), centres per class around the 8 that it sums in
registers, and iteration caps from one to more than it takes to settle."""
import numpy as np
import pytest

import jfcut
import oracle

pytestmark = pytest.mark.gpu
DTYPES = {jfcut.PIX_GRAY8: (np.uint8, 0, 255), jfcut.PIX_RGB8: (np.uint8, 0, 255),
          jfcut.PIX_I16: (np.int16, -32768, 32767)}


@pytest.mark.parametrize("pixfmt", sorted(DTYPES))
@pytest.mark.parametrize("nseeds", [2, 33, 1024, 1025, 9000, 131072, 131073, 200000])
@pytest.mark.parametrize("k_fg,k_bg,iters", [(1, 5, 1), (8, 8, 6), (9, 2, 40), (32, 32, 3)])
def test_colour_models_equal_the_restatement(ctx, pixfmt, nseeds, k_fg, k_bg, iters):
    dtype, lo, hi = DTYPES[pixfmt]
    rng = np.random.default_rng(nseeds + k_fg)
    h, w = (30, 50) if nseeds <= 1025 else (110, 100) if nseeds <= 9000 else (500, 450)
    shape = (h, w, 3) if pixfmt == jfcut.PIX_RGB8 else (h, w)
    img = rng.integers(lo, hi + 1, shape).astype(dtype)
    seeds = np.zeros(h * w, np.uint8)
    at = rng.permutation(h * w)[:nseeds]
    seeds[at] = 1 + (np.arange(nseeds) % 3 == 0)
    seeds[at[0]], seeds[at[1]] = 1, 2
    model = dict(lambda_n=100, z_weight_pct=100, lambda_t=10, k_fg=k_fg, k_bg=k_bg, seed_cap=1000000,
                 kmeans_iters=iters)
    g = jfcut.Graph(ctx, (h, w))
    g.build_from_image(img, seeds.reshape(h, w), pixfmt, model)
    e_dev, _, _ = g.state()
    e, _, _ = oracle.build_graph(img, seeds.reshape(h, w), pixfmt, model)
    assert np.array_equal(e_dev, e)
    g.close()
