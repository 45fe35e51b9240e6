"""Depths in the caller's array after a traversal that gave up at a barrier: -1
or a depth, nothing that the engine marks vertices with meanwhile."""
import ctypes

import numpy as np
import pytest

import turbobfs_gb300 as tb
from turbobfs_gb300 import graphs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lists", ["short", "long"])
@pytest.mark.parametrize("mode", ["td", "bu"])
def test_depths_after_a_timeout(gpu_available, lists, mode):
    n, fan = 20000, 4 if lists == "short" else 300
    v = np.arange(n // 2)
    src = np.concatenate([np.repeat(v[:20], fan), v[:-1]])
    dst = np.concatenate([100 + np.arange(20 * fan), v[1:]])
    h = graphs.from_edges(n, src, dst)  # directed; half of the vertices have no in-list
    P32, P64 = ctypes.POINTER(ctypes.c_int32), ctypes.POINTER(ctypes.c_int64)
    S, sg = np.full(n, 7, np.int32), np.zeros(n, np.int64)
    with tb.Graph.from_host_csc(h, keep_order=True) as g:
        o = tb.make_options(mode, True, timeout_ns=50_000_000, inject_barrier_skip=2)
        rc = tb.lib().tbfs_bfs(g.handle, 0, ctypes.byref(o), S.ctypes.data_as(P32),
                               sg.ctypes.data_as(P64), None)
        assert rc != 0
        assert S.min() == -1 and S[0] == 0
        r = g.bfs(0, mode=mode)  # the context and the graph are usable
        assert r.S[0] == 0 and r.S[1] == 1
