"""Relabel cycles run by the device (one graph launch with a loop) and by the
host (use_graph 0) give the oracle's flow and cut for every schedule kind, interval
and cap, also after a run that its sweep budget ended and after a warm edit."""
import numpy as np
import pytest

import jfcut
import oracle
from conftest import zero_boundary

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("use_graph", [0, 1])
@pytest.mark.parametrize("sched", [0, 1, 2, 3])
@pytest.mark.parametrize("interval,cap", [(1, -1), (1, 5), (3, 0), (64, 40)])
@pytest.mark.parametrize("shape", [(1, 1), (70, 210), (3, 25, 70)])
def test_cycles(ctx, shape, interval, cap, sched, use_graph):
    rng = np.random.default_rng(11 + shape[0])
    n = int(np.prod(shape))
    caps = [np.where(rng.random(n) < 0.7, rng.integers(1, 25, n), 0).astype(np.int32) for _ in range(2 * len(shape))]
    zero_boundary(shape, caps)
    e = rng.integers(-3, 3, n).astype(np.int32)
    e[rng.integers(0, n, max(1, n // 300))] -= 400
    e[rng.integers(0, n, max(1, n // 200))] += 300
    ctx.set_params(use_graph=use_graph, pr_sched=sched, relabel_interval=interval, relabel_cap=cap)
    g = jfcut.Graph(ctx, shape)
    g.set(e, caps)
    sink = int(np.maximum(-e.astype(np.int64), 0).sum())
    for turn in range(2):
        g.solve()
        flow, _, _, lab = oracle.maxflow(shape, e, caps)
        # (the oracle solves the net excess; what cs and ct of one node cancel flows too)
        assert g.flow() == flow + sink - int(np.maximum(-e.astype(np.int64), 0).sum())
        assert np.array_equal(g.labels().ravel(), lab)
        idx = np.unique(rng.integers(0, n, max(1, n // 50))).astype(np.uint32)
        add = rng.integers(1, 60, idx.size).astype(np.int32)
        g.edit_tlinks(idx, add, np.zeros(idx.size, np.int32))
        e[idx] += add
    g.close()


@pytest.mark.parametrize("use_graph", [0, 1])
@pytest.mark.parametrize("budget", [1, 2, 5])
def test_sweep_budget_ends_a_run(ctx, budget, use_graph):
    shape, n = (130, 170), 130 * 170
    rng = np.random.default_rng(3)
    caps = [rng.integers(1, 30, n).astype(np.int32) for _ in range(4)]
    zero_boundary(shape, caps)
    e = np.zeros(n, np.int32)
    e[:170] = 40
    e[-170:] = -60
    ctx.set_params(use_graph=use_graph, max_sweeps=budget, relabel_interval=1, relabel_interval_max=1)
    g = jfcut.Graph(ctx, shape)
    g.set(e, caps)
    with pytest.raises(jfcut.JfcError):
        g.solve()
    ctx.reset_params()
    ctx.set_params(use_graph=use_graph)
    g.set(e, caps)
    st = g.solve()
    flow, _, _, lab = oracle.maxflow(shape, e, caps)
    assert g.flow() == flow and np.array_equal(g.labels().ravel(), lab)
    assert st.global_relabels >= 3 and st.used_graph == use_graph
    g.close()


@pytest.mark.parametrize("interval,cap,local", [(1, 3, 1), (1, -1, 16), (2, 0, 4), (64, 40, 16)])
@pytest.mark.parametrize("shape", [(1, 1), (70, 210), (300, 333)])
def test_allocation_free_cycles(ctx, shape, interval, cap, local):
    # a run of the allocation-free solve ends after 8 cycles: short intervals need many runs
    import torch
    rng = np.random.default_rng(17 + shape[0])
    n = shape[0] * shape[1]
    caps = [np.where(rng.random(n) < 0.7, rng.integers(1, 25, n), 0).astype(np.int32) for _ in range(4)]
    zero_boundary(shape, caps)
    e = rng.integers(-3, 3, n).astype(np.int32)
    e[rng.integers(0, n, max(1, n // 300))] -= 400
    e[rng.integers(0, n, max(1, n // 200))] += 300
    params = jfcut.default_params(relabel_interval=interval, relabel_interval_max=interval, relabel_cap=cap,
                                  local_iters=local)
    d_e = torch.from_numpy(e).cuda()
    d_c = [torch.from_numpy(c).cuda() for c in caps]
    d_lab = torch.empty(n, dtype=torch.uint8, device="cuda")
    flow, _, _, lab = oracle.maxflow(shape, e, caps)
    for turn in range(2):
        d_lab.fill_(7)
        f = jfcut.solve_grid2d_noalloc(shape[1], shape[0], d_e.data_ptr(), [c.data_ptr() for c in d_c],
                                       d_lab.data_ptr(), params=params)
        assert f == flow and np.array_equal(d_lab.cpu().numpy(), lab)
