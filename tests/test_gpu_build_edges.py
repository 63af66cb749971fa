"""The capacity build against the CPU restatement, bit for bit, on widths around
the 4 pixels of a lane and the 128 of a warp, heights around its strips, rows
that start at every byte offset, and weights on both sides of a byte (tables
in shared memory or not)."""
import numpy as np
import pytest

import jfcut
import oracle

pytestmark = pytest.mark.gpu
DTYPES = {jfcut.PIX_GRAY8: (np.uint8, 0, 255), jfcut.PIX_RGB8: (np.uint8, 0, 255),
          jfcut.PIX_I16: (np.int16, -32768, 32767)}


@pytest.mark.parametrize("pixfmt", sorted(DTYPES))
@pytest.mark.parametrize("lambda_n", [100, 300])
@pytest.mark.parametrize("shape", [(2, 1), (1, 2), (3, 3), (5, 4), (17, 5), (4, 31), (16, 127), (33, 128), (2, 129),
                                   (15, 261), (2, 3, 5), (3, 17, 33), (5, 2, 130)])
def test_build_equals_the_restatement(ctx, pixfmt, lambda_n, shape):
    dtype, lo, hi = DTYPES[pixfmt]
    rng = np.random.default_rng(sum(shape) + pixfmt)
    full = shape + (3,) if pixfmt == jfcut.PIX_RGB8 else shape
    img = rng.integers(lo, hi + 1, full).astype(dtype)
    seeds = rng.choice([0, 0, 0, 1, 2], shape).astype(np.uint8)
    seeds.reshape(-1)[0], seeds.reshape(-1)[-1] = 1, 2
    model = dict(lambda_n=lambda_n, z_weight_pct=50, lambda_t=10, k_fg=3, k_bg=10, seed_cap=1000000, kmeans_iters=5)
    g = jfcut.Graph(ctx, shape)
    g.build_from_image(img, seeds, pixfmt, model)
    e_dev, r_dev, _ = g.state()
    e, caps, _ = oracle.build_graph(img, seeds, pixfmt, model)
    assert np.array_equal(e_dev, e)
    assert all(np.array_equal(r, c) for r, c in zip(r_dev, caps))
    g.close()
