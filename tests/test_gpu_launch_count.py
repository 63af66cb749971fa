"""The library's launch counter over a solve whose cycles a graph runs: every kernel
that was launched, the parts that were not due and returned at once included."""
import numpy as np
import pytest

import jfcut
import oracle
from conftest import random_grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cap", [-1, 0])
@pytest.mark.parametrize("shape,relabel,cut", [((90, 150), 1, 1), ((6, 40, 70), 4, 2)])
def test_counts_what_a_graph_launches(ctx, shape, relabel, cut, cap):
    e, caps = random_grid(shape, np.random.default_rng(4), cap_max=60, density=0.6)
    # (one run of cycles: no sweeps past the cap, one schedule)
    ctx.set_params(relabel_cap=cap, pr_sched=1)
    g = jfcut.Graph(ctx, shape)
    g.set(e, caps)
    before = jfcut.lib().jfc_kernel_launches()
    st = g.solve()
    launched = jfcut.lib().jfc_kernel_launches() - before
    assert g.flow() == oracle.maxflow(shape, e, caps)[0] and st.used_graph == 1
    # pre-push; the relabels, of which the exact one is in the graph even when the cycles' own
    # were exact; the push-relabel phases; the cut
    relabels = st.global_relabels + (1 if cap < 0 else 0)
    assert launched == 1 + relabel * relabels + st.pr_phases + cut
    g.close()
