"""Launches of the multi-instance engine on both sides of the size from which
all their instances are shared by all CTAs (2^20 vertices of the largest), with
small instances beside the large one, and a server whose launches change from
one kind to the other while queries are under way."""
import numpy as np
import pytest

import oracle
import turbobfs_gb300 as tb
from test_gpu_multi_local import GRAPHS, check
from turbobfs_gb300 import graphs

pytestmark = pytest.mark.gpu


def long_chain(n, length, fan):
    """A chain of `length` from 0 on n vertices, every vertex of it with `fan`
    vertices of its own."""
    v = np.arange(length)
    leaf = length + np.arange(length * fan)
    return graphs.from_edges(n, np.concatenate([v[:-1], np.repeat(v, fan)]),
                             np.concatenate([v[1:], leaf]))


@pytest.mark.parametrize("sigma", [True, False])
@pytest.mark.parametrize("n", [(1 << 20) - 1, 1 << 20, (1 << 20) + 1])
def test_arena_with_a_large_instance(gpu_available, n, sigma):
    names = sorted(GRAPHS)
    pick = [GRAPHS[name]() for name in names] + [(long_chain(n, 700, 5), 0)]
    want = [oracle.exact_bfs(h.col_ptr, h.row_idx, r) for h, r in pick]
    with tb.Arena([h for h, _ in pick], symmetric=False) as a:
        S, sg, stats = a.bfs([r for _, r in pick], sigma=sigma)
        S, sg = a.split(S), a.split(sg) if sigma else [None] * len(pick)
        for name, s, x, st, w in zip(names + ["large"], S, sg, stats, want):
            check(name, s, x, st, w)


def test_server_with_large_and_small_queries(gpu_available):
    hs = [long_chain((1 << 20) + 5, 3000, 3), graphs.grid(300, seed=2), graphs.grid(40, seed=3),
          long_chain(5000, 600, 4)]
    want = [oracle.exact_bfs(h.col_ptr, h.row_idx, 0) for h in hs]
    order = [1, 2, 0, 3, 2, 1, 0, 3, 2, 1]
    gs = [tb.Graph.from_host_csc(h) for h in hs]
    for i, g in enumerate(gs):  # known depths: deep ones stay in the shared launches
        g.bfs(0)
    with tb.Server(max_slots=16, mem_budget=1 << 28) as sv:
        t = [sv.submit(gs[i], 0, sigma=True) for i in order]
        for ticket, i in zip(t, order):
            r = sv.wait(ticket)[0]
            check(str(i), r.S, r.sigma, r.stats, want[i])
    for g in gs:
        g.close()
