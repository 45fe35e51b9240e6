"""Device graph building at the sizes where its passes can go wrong: lengths
around a sort tile and a compaction tile, runs of empty columns longer than a
pair fills itself, everything in the first or the last column, one digit and
several -- element for element against the host builder."""
import ctypes

import numpy as np
import pytest

import turbobfs_gb300 as tb
from turbobfs_gb300 import graphs
from turbobfs_gb300._lib import BUILD_DEDUP, BUILD_DROP_LOOPS, BUILD_SORT, BUILD_SYMMETRIZE

pytestmark = pytest.mark.gpu

FLAGS = [0, BUILD_SYMMETRIZE, BUILD_SORT, BUILD_DEDUP | BUILD_DROP_LOOPS,
         BUILD_SYMMETRIZE | BUILD_DEDUP | BUILD_DROP_LOOPS]


def edges(n, m, where, seed):
    rng = np.random.default_rng(seed)
    src = rng.integers(0, n, m)
    dst = {"any": rng.integers(0, n, m), "first": np.zeros(m), "last": np.full(m, n - 1),
           "ends": np.where(rng.random(m) < 0.5, 0, n - 1)}[where]
    return src.astype(np.int32), dst.astype(np.int32)


@pytest.mark.parametrize("where", ["any", "first", "last", "ends"])
@pytest.mark.parametrize("n,m", [(1, 3), (2, 1), (70, 4095), (66, 4096), (300, 4097), (65536, 8193),
                                 (200003, 7), (200003, 20000)])
def test_from_edges_sizes(gpu_available, n, m, where):
    src, dst = edges(n, m, where, n + m)
    for flags in FLAGS:
        want = graphs.from_edges(n, src, dst, symmetrize=bool(flags & BUILD_SYMMETRIZE),
                                 drop_loops=bool(flags & BUILD_DROP_LOOPS),
                                 dedup=bool(flags & BUILD_DEDUP), sort=bool(flags & BUILD_SORT))
        with tb.Graph.from_edges(src, dst, n, flags, keep_order=True) as g:
            cp, ic = g.csc()
        assert np.array_equal(cp, want.col_ptr) and np.array_equal(ic, want.row_idx)


@pytest.mark.parametrize("where", ["any", "first", "last", "ends"])
@pytest.mark.parametrize("n,m", [(1, 3), (66, 4097), (200003, 7), (200003, 20000)])
def test_cooc_sizes(gpu_available, n, m, where):
    src, dst = edges(n, m, where, n + 2 * m)
    order = np.argsort(dst, kind="stable")
    cp = np.concatenate([[0], np.cumsum(np.bincount(dst, minlength=n))])
    with tb.Graph.from_cooc(src, dst, n, keep_order=True) as g:
        got_cp, got_ic = g.csc()
    assert np.array_equal(got_cp, cp) and np.array_equal(got_ic, src[order])


@pytest.mark.parametrize("flip", [False, True])
def test_symmetry_is_found_or_not(gpu_available, flip):
    h = graphs.rmat(13, 8, seed=2)
    ic = h.row_idx.copy()
    if flip:  # one entry of an edge moved to another source
        ic[-1] = (ic[-1] + 1) % h.n
    with tb.Graph(h.col_ptr, ic, keep_order=True) as g:
        flags = ctypes.c_uint32()
        assert tb.lib().tbfs_graph_info(g.handle, None, None, ctypes.byref(flags)) == 0
    assert bool(flags.value & 1) == (not flip)


def test_lists_of_every_size_are_regrouped(gpu_available):
    """Renumbering copies lists by a lane, a warp or a block: a graph whose
    list lengths straddle 32 and 4096, traversed in both numberings."""
    rng = np.random.default_rng(4)
    lens = np.array([0, 1, 31, 32, 33, 127, 128, 129, 4095, 4096, 4097, 9000] + [2] * 3000)
    n = len(lens)
    src = rng.integers(0, n, lens.sum()).astype(np.int32)
    dst = np.repeat(np.arange(n), lens).astype(np.int32)
    with tb.Graph.from_edges(src, dst, n, 0) as a, tb.Graph.from_edges(src, dst, n, 0, keep_order=True) as b:
        for root in (0, 5, n - 1):
            x, y = a.bfs(root), b.bfs(root)
            assert np.array_equal(x.S, y.S) and np.array_equal(x.sigma, y.sigma)
