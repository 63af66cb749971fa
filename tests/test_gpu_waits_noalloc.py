"""A device-side wait that gives up in the allocation-free solve, which queues several
cycles behind one wait of the host: the launches behind it leave at their first
barrier, the call reports JFC_ERR_CUDA, and the next call is exact."""
import numpy as np
import pytest

import jfcut
import oracle
from conftest import random_grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile_rows", [8, 16])
def test_expired_wait_ends_an_allocation_free_call(ctx, tile_rows):
    import torch
    shape = (500, 1000)
    e, caps = random_grid(shape, np.random.default_rng(62), cap_max=80, density=0.5)
    f_ref, _, _, lab_ref = oracle.maxflow(shape, e, caps)
    d_e = torch.from_numpy(e).cuda()
    d_c = [torch.from_numpy(c).cuda() for c in caps]
    d_lab = torch.empty(e.size, dtype=torch.uint8, device="cuda")

    def solve(**kw):
        return jfcut.solve_grid2d_noalloc(shape[1], shape[0], d_e.data_ptr(), [c.data_ptr() for c in d_c],
                                          d_lab.data_ptr(), params=jfcut.default_params(tile_rows=tile_rows, **kw))

    for _ in range(2):
        with pytest.raises(jfcut.JfcError) as ei:
            solve(spin_limit=1)
        assert ei.value.code == jfcut.ERR_CUDA and "timed out" in str(ei.value)
        assert solve() == f_ref
        assert np.array_equal(d_lab.cpu().numpy(), lab_ref)
