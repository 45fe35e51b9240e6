"""Instances that one CTA runs from shared memory, against the exact oracle:
chains, levels larger than its queue and than its edges (given back to all
CTAs and taken again), vertices whose table slots are all taken, counts past
2^32 and 2^63, several instances per CTA, outputs that cannot be written in
place."""
import ctypes

import numpy as np
import pytest

import oracle
import turbobfs_gb300 as tb
from turbobfs_gb300 import graphs

pytestmark = pytest.mark.gpu


def chain(n):
    v = np.arange(n - 1)
    return graphs.from_edges(n, v, v + 1), 0


def layers(widths, k):
    """Every vertex from k consecutive ones of the layer before."""
    src, dst, first = [], [], 0
    for a, b in zip(widths, widths[1:]):
        w = np.arange(b)
        src.append(first + (np.repeat(w * a // b, k) + np.tile(np.arange(k), b)) % a)
        dst.append(first + a + np.repeat(w, k))
        first += a
    return graphs.from_edges(sum(widths), np.concatenate(src), np.concatenate(dst)), 0


def hubs(n, leaves):
    """A root, `leaves` vertices without further lists, and one behind one."""
    return graphs.from_edges(n, np.concatenate([np.zeros(leaves, np.int64), [5]]),
                             np.concatenate([1 + np.arange(leaves), [n - 1]])), 0


def crowded(n, many):
    """Two levels of vertices that share four neighbouring slots of the table."""
    ids = np.arange(2, n, dtype=np.uint64)
    slot = ((ids * 0x9E3779B1) % 2**32) >> 20
    ids = ids[(slot >= 4094) | (slot < 2)].astype(np.int64)[:2 * many]
    assert len(ids) == 2 * many
    a, b = ids[:many], ids[many:]
    src = np.concatenate([np.zeros(many, np.int64), np.repeat(a, 3), b])
    dst = np.concatenate([a, b[(np.arange(3 * many) * 7) % many], np.ones(many, np.int64)])
    return graphs.from_edges(n, src, dst), 0


GRAPHS = {
    "chain": lambda: chain(3000),
    "one_vertex": lambda: (graphs.from_edges(3, np.array([1]), np.array([2])), 0),
    "queue_edge": lambda: layers([1, 2047, 2048, 2049, 2050, 40, 1, 1, 9], 2),
    "grows_and_shrinks": lambda: layers([1, 30, 900, 27000, 9000, 300, 4, 1, 1, 300, 30000, 3], 5),
    "edges_of_a_round": lambda: layers([1, 767, 768, 769, 1, 31, 32, 33, 3071, 3072, 3073, 2], 1),
    "hub": lambda: hubs(60000, 50000),
    "small_hub": lambda: hubs(2100, 2048),
    "crowded": lambda: crowded(1 << 17, 60),
    "wide_counts": lambda: (graphs.layered_bipartite(20, 9), 0),
    "overflow": lambda: (graphs.layered_bipartite(60, 12), 0),
}


@pytest.fixture(scope="module")
def cases():
    out = []
    for name in sorted(GRAPHS):
        h, root = GRAPHS[name]()
        out.append((name, h, root, oracle.exact_bfs(h.col_ptr, h.row_idx, root)))
    return out


def check(name, S, sg, st, want):
    S0, sg0, ovf, _ = want
    assert np.array_equal(S, S0), name
    if sg is not None:
        assert np.array_equal(sg[ovf == 0], sg0[ovf == 0]), name
        assert bool(st["sigma_overflow"]) == bool(ovf.any()), name
    assert st["visited"] == (S0 >= 0).sum(), name
    assert st["levels"] == S0.max() + 1, name


@pytest.mark.parametrize("sigma", [True, False])
@pytest.mark.parametrize("copies", [1, 40])  # 40: more instances than SMs
def test_arena(gpu_available, cases, sigma, copies):
    pick = cases * copies
    with tb.Arena([c[1] for c in pick], symmetric=False) as a:
        for _ in range(2):
            S, sg, stats = a.bfs([c[2] for c in pick], sigma=sigma)
            S, sg = a.split(S), a.split(sg) if sigma else [None] * len(pick)
            for c, s, x, st in zip(pick, S, sg, stats):
                check(c[0], s, x, st, c[3])


@pytest.mark.parametrize("shift", [0, 4])  # 4: path counts not on 8 bytes
def test_device_outputs(gpu_available, cases, shift):
    import torch
    from turbobfs_gb300 import api
    with tb.Arena([c[1] for c in cases], symmetric=False) as a:
        tot = int(a.offsets[-1])
        S = torch.empty(tot, dtype=torch.int32, device="cuda")
        raw = torch.empty(8 * tot + 8, dtype=torch.uint8, device="cuda")
        o = api.make_options("td", True, outputs_on_device=True)
        roots = np.array([c[2] for c in cases], np.int32)
        tb.lib().tbfs_arena_bfs.restype = ctypes.c_int
        rc = tb.lib().tbfs_arena_bfs(a._h, roots.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)),
                                     ctypes.byref(o), S.data_ptr(), raw.data_ptr() + shift, None)
        assert rc == 0
        torch.cuda.synchronize()
        sg = raw.cpu().numpy()[shift:shift + 8 * tot].view(np.int64)
        for c, s, x in zip(cases, a.split(S.cpu().numpy()), a.split(sg)):
            S0, sg0, ovf, _ = c[3]
            assert np.array_equal(s, S0), c[0]
            assert np.array_equal(x[ovf == 0], sg0[ovf == 0]), c[0]


def test_server(gpu_available, cases):
    with tb.Server(max_slots=64, mem_budget=1 << 28) as sv:
        gs = [tb.Graph.from_host_csc(c[1]) for c in cases]
        t = [sv.submit(g, c[2], sigma=True) for _ in range(2) for g, c in zip(gs, cases)]
        for ticket, c in zip(t, cases * 2):
            r = sv.wait(ticket)[0]
            check(c[0], r.S, r.sigma, r.stats, c[3])
        for g in gs:
            g.close()
