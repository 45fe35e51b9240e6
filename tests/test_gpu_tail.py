"""A dense core with a long thin tail: a traversal with path counts that went
bottom-up in the core must not stay so along the tail, where every bottom-up
level reads the depths of all vertices."""
import numpy as np
import pytest

import oracle
import turbobfs_gb300 as tb
from turbobfs_gb300 import graphs

pytestmark = pytest.mark.gpu


def core_and_chain(n, tail, lists):
    """A random core of 2^15 vertices (hubs, or lists of about 20), a chain of `tail`
    behind it, the other vertices alone."""
    rng = np.random.default_rng(7)
    nc = 1 << 15
    if lists == "hubs":
        u = (nc * rng.random(nc * 16) ** 6).astype(np.int64)
        v = rng.integers(0, nc, nc * 16)
    else:
        u, v = rng.integers(0, nc, nc * 10), rng.integers(0, nc, nc * 10)
    c = nc + np.arange(tail - 1)
    return graphs.from_edges(n, np.concatenate([u, [1], c]), np.concatenate([v, [nc], c + 1]),
                             symmetrize=True, drop_loops=True, dedup=True)


@pytest.mark.parametrize("lists", ["hubs", "short"])
@pytest.mark.parametrize("n", [1 << 20, 1 << 22])
def test_tail_is_not_scanned(gpu_available, n, lists):
    h = core_and_chain(n, 1500, lists)
    S0, sg0, ovf, levels = oracle.exact_bfs(h.col_ptr, h.row_idx, 2)
    assert levels > 1500
    with tb.Graph.from_host_csc(h) as g:
        r = g.bfs(2)
        assert np.array_equal(r.S, S0)
        assert np.array_equal(r.sigma[ovf == 0], sg0[ovf == 0])
        # a few levels of the core, and of the tail until they cost what a change does
        assert 1 <= r.stats["bu_levels"] <= 12
