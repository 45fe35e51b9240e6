"""Push levels of a batch whose counts are added along the level's own edges:
the new vertices are finished, with counts of 0, in a phase before, one to
several rounds of them per item, for every row width, against the exact
oracle."""
import numpy as np
import pytest

import oracle
import turbobfs_gb300 as tb
from turbobfs_gb300 import graphs

pytestmark = pytest.mark.gpu


def wide_fan(fan, out, feeders):
    """0 and 1 -> fan vertices, each with `out` edges into a second layer of
    fan // 3, and `feeders` vertices that nothing leads to with an edge to each of
    the fan's first: long in-lists there, few edges that find them."""
    v = 2 + np.arange(fan)
    second = 2 + fan + np.arange(fan // 3)
    rng = np.random.default_rng(fan)
    feed = 2 + fan + fan // 3 + np.arange(feeders)
    src = [np.zeros(fan, np.int64), np.ones(fan // 2, np.int64), np.repeat(v, out),
           np.repeat(feed, 40)]
    dst = [v, v[:fan // 2], second[rng.integers(0, fan // 3, fan * out)],
           np.tile(v[:40], feeders)]
    return graphs.from_edges(2 + fan + fan // 3 + feeders, np.concatenate(src), np.concatenate(dst))


@pytest.mark.parametrize("k", [2, 33, 70, 200])  # rows of 1, 2, 4 and 8 words
@pytest.mark.parametrize("fan", [50, 1000, 30000, 130000])
def test_counts_along_edges(gpu_available, fan, k):
    h = wide_fan(fan, 12, 3000)
    rng = np.random.default_rng(k)
    roots = np.concatenate([[0, 1], rng.integers(0, h.n, k - 2)]).astype(np.int32)
    pick = [0, 1] + list(range(2, k, 13))
    want = {i: oracle.exact_bfs(h.col_ptr, h.row_idx, int(roots[i])) for i in pick}
    with tb.Graph.from_host_csc(h) as g:
        for mode in ("td", "auto"):
            S, sg, stats = g.bfs_batch(roots, mode=mode)
            for i in pick:
                S0, sg0, _, _ = want[i]
                assert np.array_equal(S[i], S0) and np.array_equal(sg[i], sg0)
                assert stats[i]["visited"] == (S0 >= 0).sum()
