"""Capacity tables (n-link weight over the contrast, t-link cost over the
quantised probability) against the CPU restatement, bit for bit: they are
found by their runs of equal entries, so the cases are those where runs are
shortest and longest — scales from 1 to more than the table has entries, an
image without contrast (one run), and one with two grey levels only."""
import numpy as np
import pytest

import jfcut
import oracle

pytestmark = pytest.mark.gpu
DTYPES = {jfcut.PIX_GRAY8: (np.uint8, 0, 255), jfcut.PIX_RGB8: (np.uint8, 0, 255),
          jfcut.PIX_I16: (np.int16, -32768, 32767)}


@pytest.mark.parametrize("pixfmt", sorted(DTYPES))
@pytest.mark.parametrize("lambda_n,lambda_t", [(1, 1), (100, 10), (7, 5000), (300000, 1000000)])
@pytest.mark.parametrize("content", ["noise", "flat", "two_level"])
def test_tables_equal_the_restatement(ctx, pixfmt, lambda_n, lambda_t, content):
    dtype, lo, hi = DTYPES[pixfmt]
    rng = np.random.default_rng(lambda_n + pixfmt)
    h, w = 45, 70
    shape = (h, w, 3) if pixfmt == jfcut.PIX_RGB8 else (h, w)
    if content == "noise":
        img = rng.integers(lo, hi + 1, shape).astype(dtype)
    elif content == "flat":
        img = np.full(shape, 17, dtype)
    else:
        img = np.where(rng.random(shape) < 0.5, lo, hi).astype(dtype)
    seeds = np.zeros((h, w), np.uint8)
    seeds[5, 3:40] = 1
    seeds[40, 20:66] = 2
    model = dict(lambda_n=lambda_n, z_weight_pct=100, lambda_t=lambda_t, k_fg=3, k_bg=4, seed_cap=1000000,
                 kmeans_iters=8)
    g = jfcut.Graph(ctx, (h, w))
    g.build_from_image(img, seeds, pixfmt, model)
    e_dev, r_dev, _ = g.state()
    e, caps, _ = oracle.build_graph(img, seeds, pixfmt, model)
    assert np.array_equal(e_dev, e)
    assert all(np.array_equal(r, c) for r, c in zip(r_dev, caps))
    g.close()
