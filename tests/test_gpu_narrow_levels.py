"""Narrow levels (vertices kept in shared memory) against the exact oracle.

Graphs whose out-lists hold at most 64 entries, at the sizes where the narrow
levels can go wrong: chains (one vertex a level), even shares every 32 levels,
a CTA with more than 64 and more than 256 finds in a level, levels that grow
beyond what is narrow and shrink again, directed lists, counts past 2^63 (also
bottom-up, where parents are found by their depth then).
"""
import numpy as np
import pytest

import oracle
import turbobfs_gb300 as tb
from turbobfs_gb300 import graphs

pytestmark = pytest.mark.gpu


def _both(a, b):
    return np.concatenate([a, b]), np.concatenate([b, a])


def _chain(n):
    v = np.arange(n - 1)
    return n, *_both(v, v + 1), 0


def _grid(w, h):
    v = np.arange(w * h).reshape(h, w)
    a = np.concatenate([v[:, :-1].ravel(), v[:-1].ravel()])
    b = np.concatenate([v[:, 1:].ravel(), v[1:].ravel()])
    return w * h, *_both(a, b), (h // 2) * w + w // 2


def _tree(fan, depth, tail):
    """A full tree, whose leaves all lead into one chain."""
    n, level, a, b = 1, [0], [], []
    for _ in range(depth):
        nxt = []
        for v in level:
            for _ in range(fan):
                a.append(v)
                b.append(n)
                nxt.append(n)
                n += 1
        level = nxt
    # leaves into ever fewer vertices, 8 at a time, so that lists stay short
    while len(level) > 1:
        nxt = list(range(n, n + (len(level) + 7) // 8))
        a += level
        b += [nxt[i // 8] for i in range(len(level))]
        n += len(nxt)
        level = nxt
    for _ in range(tail):
        a.append(level[0])
        b.append(n)
        level = [n]
        n += 1
    return n, np.array(a), np.array(b), 0


def _diamonds(k):
    """k diamonds in a row: 2^k paths to the last vertex."""
    a, b = [], []
    for i in range(k):
        v = 3 * i
        a += [v, v, v + 1, v + 2]
        b += [v + 1, v + 2, v + 3, v + 3]
    return 3 * k + 1, np.array(a), np.array(b), 0


def _random(n, degree, seed):
    """n * degree random edges, of which every vertex keeps at most 64."""
    rng = np.random.default_rng(seed)
    a, b = rng.integers(0, n, n * degree), rng.integers(0, n, n * degree)
    order = np.argsort(a, kind="stable")
    a, b = a[order], b[order]
    rank = np.arange(len(a)) - np.searchsorted(a, a)
    return n, a[rank < 64], b[rank < 64], 0


GRAPHS = {
    "random_1000_of_7": lambda: _random(1000, 7, 1),
    "random_3000_of_60": lambda: _random(3000, 60, 2),
    "random_30000_of_9": lambda: _random(30000, 9, 3),
    "tree_64_fan": lambda: _tree(64, 2, 40),
    "tree_65_fan": lambda: _tree(65, 2, 40),
    "chain_700": lambda: _chain(700),
    "strip_3x400": lambda: _grid(3, 400),
    "grid_150x140": lambda: _grid(150, 140),
    "tree_16_fan": lambda: _tree(16, 2, 40),
    "tree_2_fan": lambda: _tree(2, 15, 70),
    "tree_12_fan": lambda: _tree(12, 4, 5),
    "diamonds_62": lambda: _diamonds(62),
    "diamonds_63": lambda: _diamonds(63),
    "diamonds_130": lambda: _diamonds(130),
}


@pytest.mark.parametrize("mode", ["auto", "td", "bu"])
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_narrow_levels(gpu_available, name, mode):
    n, src, dst, root = GRAPHS[name]()
    h = graphs.from_edges(n, src, dst)
    S, sg, ovf, _ = oracle.exact_bfs(h.col_ptr, h.row_idx, root)
    sizes = np.bincount(S[S >= 0])
    with tb.Graph.from_host_csc(h) as g:
        for units in (None, 1):
            r = g.bfs(root, mode=mode, ctas_per_sm=units)
            assert np.array_equal(r.S, S)
            assert np.array_equal(r.sigma[ovf == 0], sg[ovf == 0])
            assert bool(r.stats["sigma_overflow"]) == bool(ovf.any())
            assert r.stats["levels"] == len(sizes)
            assert r.stats["visited"] == sizes.sum()
            r = g.bfs(root, mode=mode, sigma=False, ctas_per_sm=units, trace=1024)
            assert np.array_equal(r.S, S)
            assert [t["vertices"] for t in r.stats["trace"]] == sizes.tolist()
