"""Capacity tables at scales where a weight or cost leaves 32 bits (it becomes the
lowest int, as the restatement's conversion gives it): such a table is not
taken for one of small entries."""
import numpy as np
import pytest

import jfcut
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pixfmt", [jfcut.PIX_GRAY8, jfcut.PIX_RGB8, jfcut.PIX_I16])
@pytest.mark.parametrize("shape,lambda_n,z_weight_pct,lambda_t", [
    ((45, 70), 100, 100, 200_000_000), ((45, 70), 100, 100, 2_147_483_647), ((6, 20, 45), 100, 100, 200_000_000),
    ((6, 20, 45), 200, 2_000_000_000, 10), ((45, 70), 255, 100, 21), ((45, 70), 255, 100, 22), ((45, 70), 256, 100, 21)])
def test_entries_past_32_bits(ctx, shape, lambda_n, z_weight_pct, lambda_t, pixfmt):
    rng = np.random.default_rng(lambda_n + pixfmt)
    lo, hi, dtype = (-32768, 32767, np.int16) if pixfmt == jfcut.PIX_I16 else (0, 255, np.uint8)
    img = rng.integers(lo, hi + 1, shape + ((3,) if pixfmt == jfcut.PIX_RGB8 else ())).astype(dtype)
    seeds = np.zeros(shape, np.uint8)
    seeds[..., 5, 3:40] = 1
    seeds[..., -4, 20:44] = 2
    model = dict(lambda_n=lambda_n, z_weight_pct=z_weight_pct, lambda_t=lambda_t, k_fg=3, k_bg=4, seed_cap=1000000,
                 kmeans_iters=8)
    g = jfcut.Graph(ctx, shape)
    g.build_from_image(img, seeds, pixfmt, model)
    e_dev, r_dev, _ = g.state()
    e, caps, _ = oracle.build_graph(img, seeds, pixfmt, model)
    assert np.array_equal(e_dev.ravel(), e)
    assert all(np.array_equal(r.ravel(), c) for r, c in zip(r_dev, caps))
    g.close()
