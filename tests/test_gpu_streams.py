"""Work that is ordered by the library alone, whatever stream the caller uses:
a graph's creation leaves nothing queued that a traversal on a non-blocking
stream would have to wait for."""
import numpy as np
import pytest

import oracle
import turbobfs_gb300 as tb
from turbobfs_gb300 import graphs

pytestmark = pytest.mark.gpu


def star(n, leaves):
    """A list long enough for hub segments on n vertices (the tables of creation
    are filled by passes over all of them)."""
    return graphs.from_edges(n, np.zeros(leaves, np.int64), 1 + np.arange(leaves),
                             symmetrize=True)


@pytest.mark.parametrize("make", ["csc", "cooc", "edges"])
def test_creation_leaves_nothing_pending(gpu_available, make):
    import torch
    legacy = torch.cuda.default_stream()
    n, leaves = 1 << 24, 3000
    zero, leaf = np.zeros(leaves, np.int32), (1 + np.arange(leaves)).astype(np.int32)
    h = star(n, leaves)
    for _ in range(3):
        legacy.synchronize()
        if make == "csc":
            g = tb.Graph.from_host_csc(h)
        elif make == "cooc":
            g = tb.Graph.from_cooc(np.concatenate([zero, leaf]), np.concatenate([leaf, zero]), n)
        else:
            g = tb.Graph.from_edges(zero, leaf, n, graphs.BUILD_SYMMETRIZE)
        idle = legacy.query()
        g.close()
        assert idle


def test_first_traversal_on_a_side_stream(gpu_available):
    import torch
    h = star(1 << 20, 5000)
    S0, sg0, _, _ = oracle.exact_bfs(h.col_ptr, h.row_idx, 1)
    side = torch.cuda.Stream()
    for mode in ("auto", "bu"):
        g = tb.Graph.from_host_csc(h)
        r = g.bfs(1, mode=mode, stream=side.cuda_stream)
        g.close()
        assert np.array_equal(r.S, S0) and np.array_equal(r.sigma, sg0)
