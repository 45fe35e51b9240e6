"""Bottom-up levels with path counts (one pass finds and counts): in-list
lengths at the edges of the schedule's classes, counts past 20 and 64 bits,
items of equal cost and of plain words, every start of a list in its group --
against the exact oracle."""
import numpy as np
import pytest

import oracle
import turbobfs_gb300 as tb
from turbobfs_gb300 import graphs

pytestmark = pytest.mark.gpu


def fan(lens, mids, seed):
    """Root 0 -> `mids` vertices -> one vertex per entry of lens with that many
    in-list entries (repeats allowed) from the middle, then a last vertex fed
    by all of those; directed, with two unreachable vertices at the end."""
    rng = np.random.default_rng(seed)
    lens = np.asarray(lens)
    first = 1 + mids
    src = [np.zeros(mids, np.int64)]
    dst = [np.arange(1, first)]
    src.append(rng.integers(1, first, int(lens.sum())))
    dst.append(np.repeat(first + np.arange(len(lens)), lens))
    last = first + len(lens)
    src.append(first + np.arange(len(lens)))
    dst.append(np.full(len(lens), last))
    src.append(np.array([last + 2]))
    dst.append(np.array([last + 1]))
    return graphs.from_edges(last + 3, np.concatenate(src), np.concatenate(dst))


def check(h, root, **kw):
    S, sg, ovf, _ = oracle.exact_bfs(h.col_ptr, h.row_idx, root)
    for keep in (False, True):
        with tb.Graph.from_host_csc(h, keep_order=keep) as g:
            for mode in ("bu", "auto"):
                res = g.bfs(root, mode=mode, **kw)
                assert np.array_equal(res.S, S)
                assert np.array_equal(res.sigma[ovf == 0], sg[ovf == 0])
                assert bool(res.stats["sigma_overflow"]) == bool(ovf.any())


EDGES = [1, 2, 7, 8, 9, 10, 47, 48, 49, 50, 127, 128, 129, 177, 1023, 1024, 1025, 2048, 2049, 5000]


@pytest.mark.parametrize("lens", [[x] for x in EDGES] + [EDGES, EDGES * 7, [3] * 200, [30] * 130])
def test_list_lengths(gpu_available, lens):
    check(fan(lens, 700, len(lens)), 0)


@pytest.mark.parametrize("n", [31, 32, 33, 127, 128, 129, 1000])
def test_group_edges(gpu_available, n):
    check(fan(np.arange(n) % 60 + 1, 257, n), 0)


@pytest.mark.parametrize("width,layers", [(3, 12), (20, 6), (60, 11), (16, 17)])
def test_large_counts(gpu_available, width, layers):
    # width ** (layers - 1) paths: past 2**20, past 2**32 and past 2**63
    check(graphs.layered_bipartite(width, layers), 0)


@pytest.mark.parametrize("alpha", [0.01, 1e6])
def test_heavy_levels(gpu_available, alpha):
    h = graphs.rmat(16, 24, seed=9)
    check(h, int(graphs.pick_roots(h, 1, seed=9)[0]), alpha=alpha)
