"""Batch levels cut into items of different sizes, against the exact oracle:
one to a few edges, a handful of vertices for all warps, runs of empty lists
between the owners of neighbouring edges, hubs, counts added along a push
level's own edges (past 2^32 and 2^63 too), and every row width."""
import numpy as np
import pytest

import oracle
import turbobfs_gb300 as tb
from turbobfs_gb300 import graphs

pytestmark = pytest.mark.gpu


def sparse(n, m, seed):
    """Directed: most vertices have no out-list."""
    rng = np.random.default_rng(seed)
    few = rng.choice(n, n // 40 + 1, replace=False)
    return graphs.from_edges(n, rng.choice(few, m), rng.integers(0, n, m))


def fan_of_leaves(fan):
    """0 -> fan vertices, of which the first and the last lead on."""
    v = 1 + np.arange(fan)
    return graphs.from_edges(fan + 3, np.concatenate([np.zeros(fan, np.int64), [1, fan]]),
                             np.concatenate([v, [fan + 1, fan + 2]]))


def fed_diamonds(k, feeders):
    """k diamonds in a row, 2^k paths, and into each vertex an edge from every
    one of `feeders` vertices that nothing leads to: few edges per level, long
    in-lists."""
    n = 3 * k + 1
    v = 3 * np.arange(k)
    src = [v, v, v + 1, v + 2, n + np.tile(np.arange(feeders), n)]
    dst = [v + 1, v + 2, v + 3, v + 3, np.repeat(np.arange(n), feeders)]
    return graphs.from_edges(n + feeders, np.concatenate(src), np.concatenate(dst))


GRAPHS = {
    "fed_diamonds_20": lambda: fed_diamonds(20, 300),
    "fed_diamonds_70": lambda: fed_diamonds(70, 300),
    "chain": lambda: graphs.from_edges(70, np.arange(69), 1 + np.arange(69)),
    "sparse_lists": lambda: sparse(5000, 9000, 1),
    "leaves_31": lambda: fan_of_leaves(31),
    "leaves_32": lambda: fan_of_leaves(32),
    "leaves_33": lambda: fan_of_leaves(33),
    "leaves_9000": lambda: fan_of_leaves(9000),
    "grid_40": lambda: graphs.grid(40, seed=3),
    "rmat_11": lambda: graphs.rmat(11, 16, seed=4),
    "layers": lambda: graphs.layered_bipartite(33, 7),
}


@pytest.mark.parametrize("k", [1, 33, 70, 200])  # rows of 1, 2, 4 and 8 words
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_items(gpu_available, name, k):
    h = GRAPHS[name]()
    rng = np.random.default_rng(k)
    roots = np.concatenate([[0], rng.integers(0, h.n, k - 1)]).astype(np.int32)
    want = {int(r): oracle.exact_bfs(h.col_ptr, h.row_idx, int(r)) for r in set(roots.tolist())}
    with tb.Graph.from_host_csc(h) as g:
        for mode in ("td", "bu", "auto"):
            for sigma in (True, False):
                S, sg, stats = g.bfs_batch(roots, mode=mode, sigma=sigma)
                for i, r in enumerate(roots.tolist()):
                    S0, sg0, ovf, _ = want[r]
                    assert np.array_equal(S[i], S0)
                    assert stats[i]["visited"] == (S0 >= 0).sum()
                    if sigma:
                        assert np.array_equal(sg[i][ovf == 0], sg0[ovf == 0])
                        assert bool(stats[i]["sigma_overflow"]) == bool(ovf.any())
