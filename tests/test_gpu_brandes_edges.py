"""Betweenness at the edges of the sweep's list classes and groups, and on
graphs too deep for the six-class sort or for shared-memory counters at all:
bit-exact against the oracle's summation order."""
import numpy as np
import pytest

import oracle
import turbobfs_gb300 as tb
from turbobfs_gb300 import graphs

pytestmark = pytest.mark.gpu


def spokes(lens, seed):
    """Vertices with the given degrees, joined to a pool of others; the pool
    is a ring, so everything is connected."""
    rng = np.random.default_rng(seed)
    pool = max(4000, max(lens) + 1)
    src = [np.repeat(np.arange(len(lens)), lens), len(lens) + np.arange(pool)]
    dst = [len(lens) + np.concatenate([rng.choice(pool, x, replace=False) for x in lens]),
           len(lens) + (np.arange(pool) + 1) % pool]
    return graphs.from_edges(len(lens) + pool, np.concatenate(src), np.concatenate(dst),
                             symmetrize=True)


def path(n):
    v = np.arange(n - 1)
    # a chord every 50 vertices, so that some counts exceed one
    c = np.arange(0, n - 3, 50)
    return graphs.from_edges(n, np.concatenate([v, c]), np.concatenate([v + 1, c + 2]), symmetrize=True)


CASES = {
    "short": lambda: spokes([1, 3, 4, 7, 8, 15, 16, 31] * 5, 1),
    "edges": lambda: spokes([31, 32, 33, 63, 64, 65, 127, 255, 256, 257, 2047, 2048, 2049, 4097], 2),
    "one group": lambda: spokes([40] * 8, 3),
    "odd group": lambda: spokes([40] * 9 + [300] * 3, 4),
    "many lists": lambda: spokes([33] * 700, 5),
    "deep 1800": lambda: path(1800),
    "deep 1900": lambda: path(1900),  # more keys than fit with six classes
    "deep 4000": lambda: path(4000),  # ... and with three
}


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("k", [1, 5, 33])
def test_brandes_edges(gpu_available, name, k):
    h = CASES[name]()
    roots = np.random.default_rng(k).integers(0, h.n, k).astype(np.int32)
    roots[0] = 0
    want, wovf = oracle.brandes(h.col_ptr, h.row_idx, roots)
    for keep in (False, True):
        with tb.Graph.from_host_csc(h, keep_order=keep) as g:
            bc, ovf = g.betweenness(roots)
        assert ovf == wovf
        assert np.array_equal(bc, want)
