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


@pytest.mark.parametrize("sigma", [True, False])
def test_arena_beside_other_kernels(gpu_available, sigma):
    """CTAs of a launch that start at different times: matrix products on another
    stream hold SMs while arenas of instances that are done in one to a few
    levels, and of some that are not, are traversed."""
    import torch
    rng = np.random.default_rng(5)
    hs, roots = [], []
    for i in range(400):
        if i % 40 == 39:
            h = graphs.grid(48, seed=i)
        else:
            n = int(rng.integers(1, 40))
            m = int(rng.integers(0, 2 * n))
            h = graphs.from_edges(n, rng.integers(0, n, m), rng.integers(0, n, m), symmetrize=True)
        hs.append(h)
        roots.append(int(rng.integers(0, h.n)))
    want = [oracle.exact_bfs(h.col_ptr, h.row_idx, r) for h, r in zip(hs, roots)]
    side = torch.cuda.Stream()
    a_mat = torch.ones(4096, 4096, dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    with tb.Arena(hs) as a:
        for _ in range(20):
            with torch.cuda.stream(side):
                for _ in range(60):
                    torch.mm(a_mat, a_mat)
            S, sg, stats = a.bfs(roots, sigma=sigma)
            sg = a.split(sg) if sigma else [None] * len(hs)
            for s, x, st, (S0, sg0, ovf, levels) in zip(a.split(S), sg, stats, want):
                assert np.array_equal(s, S0)
                assert x is None or np.array_equal(x[ovf == 0], sg0[ovf == 0])
                assert st["levels"] == levels and st["visited"] == (S0 >= 0).sum()
    side.synchronize()
