"""Push levels of a batch whose counts are added along the level's own edges: the
new vertices' counts start at 0, written with the discovery at the first level
and in a phase of its own (one to several rounds of vertices per item) at later
ones, for every row width, against the exact oracle."""
import numpy as np
import pytest

import oracle
import turbobfs_gb300 as tb
from turbobfs_gb300 import graphs

pytestmark = pytest.mark.gpu


def wide_fan(fan, out, feeders):
    """2 -> 0 and 1 -> fan vertices, each with `out` edges into a second layer of
    fan // 3, and `feeders` vertices that nothing leads to with an edge to each of
    the fan's first: long in-lists there, few edges that find them."""
    v = 3 + np.arange(fan)
    second = 3 + fan + np.arange(fan // 3)
    rng = np.random.default_rng(fan)
    feed = 3 + fan + fan // 3 + np.arange(feeders)
    src = [np.array([2, 2]), np.zeros(fan, np.int64), np.ones(fan // 2, np.int64),
           np.repeat(v, out), np.repeat(feed, 40)]
    dst = [np.array([0, 1]), v, v[:fan // 2], second[rng.integers(0, fan // 3, fan * out)],
           np.tile(v[:40], feeders)]
    return graphs.from_edges(3 + fan + fan // 3 + feeders, np.concatenate(src), np.concatenate(dst))


@pytest.mark.parametrize("k", [3, 33, 70, 200])  # rows of 1, 2, 4 and 8 words
@pytest.mark.parametrize("fan", [50, 1000, 30000, 130000])
@pytest.mark.parametrize("level", ["first", "later"])
def test_counts_along_edges(gpu_available, level, fan, k):
    h = wide_fan(fan, 12, 3000)
    rng = np.random.default_rng(k)
    if level == "first":
        roots = np.concatenate([[0, 1, 2], rng.integers(0, h.n, k - 3)])
    else:  # the others lead nowhere: the fan is found at the second level
        roots = np.concatenate([[2, 2, 2], 3 + fan + rng.integers(0, fan // 3, k - 3)])
    roots = roots.astype(np.int32)
    pick = [0, 1, 2] + list(range(3, k, 13))
    want = {i: oracle.exact_bfs(h.col_ptr, h.row_idx, int(roots[i])) for i in pick}
    with tb.Graph.from_host_csc(h) as g:
        for mode in ("td", "auto"):
            S, sg, stats = g.bfs_batch(roots, mode=mode)
            for i in pick:
                S0, sg0, _, _ = want[i]
                assert np.array_equal(S[i], S0) and np.array_equal(sg[i], sg0)
                assert stats[i]["visited"] == (S0 >= 0).sum()
