"""Performance cases of the BFS framework: the calls a user's program makes,
through the public entry points (the C ABI of include/tbfs.h and
include/tbfs_compat.h, called through the package's ctypes binding, and the
package's own classes), over the range of sizes, graph families and options
they are used with.

Kinds of case
  bfs      one traversal of a resident graph, S (+ sigma) into device memory
  fresh    a graph built from an edge list on the device, traversed once and
           dropped
  batch    many roots of one resident graph in one frontier-matrix call
  arena    many small graphs packed together, one root each, one call
  serve    a burst of queries to the serving loop, answers in host memory
  dropin   the reference's entry points: host arrays in, host arrays out
  brandes  betweenness of a set of roots

Families of graph: "rmat" (a/b/c/d = .57/.19/.19/.05, vertices permuted, no
self-loops or repeats), "er" (uniform random edges) and "grid" (side x side,
a tenth of the edges deleted, 1 % chords within Manhattan distance 8).  All
are generated on the GPU from the seed alone.
"""
import ctypes
import math

import numpy as np
import torch

import turbobfs_gb300 as tb

SYMMETRIC, DEVICE_PTRS = 0x1, 0x2                   # TBFS_GRAPH_*
SYMMETRIZE, DROP_LOOPS, DEDUP = 0x1, 0x2, 0x4       # TBFS_BUILD_*
ROOT_MAJOR, VERTEX_MAJOR = 0, 1                     # TBFS_LAYOUT_*
DEV = "cuda"
_I32P = ctypes.POINTER(ctypes.c_int32)
_I64P = ctypes.POINTER(ctypes.c_int64)


# ------------------------------------------------------------------ cases ---

def listed():
    return [
        # the smallest call: latency of one query on a small graph (the plain
        # Erdos-Renyi configuration, n = 4096, average degree 8)
        {"name": "bfs_er4k", "kind": "bfs", "family": "er", "n": 4096, "degree": 8, "sigma": True, "mode": "auto"},
        # an ordinary query on a social-network-like graph of odd size
        {"name": "bfs_rmat100k", "kind": "bfs", "family": "rmat", "n": 100003, "degree": 32, "sigma": True, "mode": "auto"},
        # reachability and distances only, no path counts, on a graph without hubs
        {"name": "depths_er1m", "kind": "bfs", "family": "er", "n": 1000003, "degree": 16, "sigma": False, "mode": "auto"},
        # the headline: direction-optimizing BFS with path counts, RMAT scale 22
        {"name": "bfs_rmat22", "kind": "bfs", "family": "rmat", "n": 1 << 22, "degree": 32, "sigma": True, "mode": "auto"},
        # road-like graph, thousands of small levels
        {"name": "bfs_grid2048", "kind": "bfs", "family": "grid", "n": 2048 * 2048, "degree": 4, "sigma": True, "mode": "auto"},
        # a directed graph that arrives as an edge list, is traversed once and dropped
        {"name": "fresh_directed512k", "kind": "fresh", "family": "rmat", "n": 1 << 19, "degree": 32, "undirected": False, "sigma": True},
        # 256 roots with path counts, the forward half of a centrality run
        {"name": "batch_rmat20_256", "kind": "batch", "family": "rmat", "n": 1 << 20, "degree": 32, "k": 256, "sigma": True, "layout": ROOT_MAJOR},
        # landmark distances: a few dozen roots, depths only, one row per vertex
        {"name": "batch_rmat200k_40", "kind": "batch", "family": "rmat", "n": 200001, "degree": 24, "k": 40, "sigma": False, "layout": VERTEX_MAJOR},
        # a data set of many small graphs, one root each
        {"name": "arena_mixed192", "kind": "arena", "graphs": 192, "lo": 10, "hi": 18, "sigma": True},
        # a burst of queries over resident graphs of mixed families and sizes
        {"name": "serve_mixed28", "kind": "serve", "graphs": 14, "lo": 12, "hi": 18, "queries": 28, "sigma": True},
        # what the reference's main program does: host CSC in, S and sigma out
        {"name": "dropin_tdbu_rmat20", "kind": "dropin", "entry": "tdbu", "family": "rmat", "n": 1 << 20, "degree": 32},
        # betweenness from a sample of roots
        {"name": "brandes_rmat18_16", "kind": "brandes", "family": "rmat", "n": 1 << 18, "degree": 32, "k": 16},
    ]


def _size(rng, lo, hi):
    return int(round(2.0 ** rng.uniform(lo, hi)))


def draw(rng):
    kind = rng.choice(["bfs", "bfs", "bfs", "fresh", "batch", "arena", "serve", "dropin", "brandes"])
    family = rng.choice(["rmat", "rmat", "er", "grid"])
    degree = rng.randint(6, 40)
    if kind == "bfs":
        sigma = rng.random() < 0.75
        mode = "auto"
        if family == "grid":
            side = int(2.0 ** rng.uniform(5, 11))
            return {"kind": kind, "family": family, "n": side * side, "degree": 4, "sigma": sigma, "mode": mode}
        if rng.random() < 0.25:
            mode = rng.choice(["td", "bu"])
        top = 21.5 if mode == "auto" else 18
        return {"kind": kind, "family": family, "n": _size(rng, 10, top), "degree": degree, "sigma": sigma, "mode": mode}
    if kind == "fresh":
        if family == "grid":
            family = "er"
        return {"kind": kind, "family": family, "n": _size(rng, 12, 20), "degree": degree,
                "undirected": rng.random() < 0.5, "sigma": rng.random() < 0.75}
    if kind == "batch":
        if family == "grid":
            side = int(2.0 ** rng.uniform(5, 8))
            n, degree = side * side, 4
        else:
            n = _size(rng, 11, 18.5)
        return {"kind": kind, "family": family, "n": n, "degree": degree, "k": rng.randint(2, 256),
                "sigma": rng.random() < 0.7, "layout": rng.choice([ROOT_MAJOR, VERTEX_MAJOR])}
    if kind == "arena":
        return {"kind": kind, "graphs": rng.randint(3, 160), "lo": 10, "hi": rng.randint(12, 17), "sigma": rng.random() < 0.75}
    if kind == "serve":
        return {"kind": kind, "graphs": rng.randint(3, 14), "lo": 12, "hi": rng.randint(13, 18),
                "queries": rng.randint(4, 30), "sigma": rng.random() < 0.75}
    if kind == "dropin":
        if family == "grid":
            side = int(2.0 ** rng.uniform(5, 9.5))
            n, degree = side * side, 4
        else:
            n = _size(rng, 11, 20)
        return {"kind": kind, "entry": rng.choice(["td", "bu", "tdbu", "cooc"]), "family": family, "n": n, "degree": degree}
    if family == "grid":
        side = int(2.0 ** rng.uniform(5, 7.5))
        n, degree = side * side, 4
    else:
        n = _size(rng, 10, 18)
    return {"kind": kind, "family": family, "n": n, "degree": degree, "k": rng.randint(1, 24)}


# ----------------------------------------------------------------- graphs ---

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _rmat_edges(n, m, g):
    u = torch.zeros(m, dtype=torch.int32, device=DEV)
    v = torch.zeros(m, dtype=torch.int32, device=DEV)
    for _ in range(max(1, (n - 1).bit_length())):
        r = torch.rand(m, generator=g, device=DEV)
        ub = r >= 0.76
        vb = ((r >= 0.57) & ~ub) | (r >= 0.95)
        u = u * 2 + ub
        v = v * 2 + vb
    perm = torch.randperm(n, generator=g, device=DEV)
    return perm[(u % n).long()], perm[(v % n).long()]


def _er_edges(n, m, g):
    return (torch.randint(n, (m,), generator=g, device=DEV), torch.randint(n, (m,), generator=g, device=DEV))


def _grid_edges(side, g):
    n = side * side
    at = torch.arange(n, device=DEV)
    x, y = at % side, at // side
    u = torch.cat([at[x < side - 1], at[y < side - 1]])
    v = torch.cat([at[x < side - 1] + 1, at[y < side - 1] + side])
    keep = torch.rand(u.numel(), generator=g, device=DEV) >= 0.10
    u, v = u[keep], v[keep]
    # chords: at most one from and one to a vertex, so degrees stay <= 6
    c = max(1, n // 100)
    cu = torch.randperm(n, generator=g, device=DEV)[:c]
    dx = torch.randint(-4, 5, (c,), generator=g, device=DEV)
    dy = torch.randint(-4, 5, (c,), generator=g, device=DEV)
    cv = (cu // side + dy).clamp(0, side - 1) * side + (cu % side + dx).clamp(0, side - 1)
    first = torch.full((n,), c, dtype=torch.long, device=DEV)
    first.scatter_reduce_(0, cv, torch.arange(c, device=DEV), "amin")
    one = first[cv] == torch.arange(c, device=DEV)
    return torch.cat([u, cu[one]]), torch.cat([v, cv[one]])


def _edges(family, n, degree, g):
    """Directed edge list (u -> v), each undirected edge once, repeats and
    self-loops still in it."""
    if family == "grid":
        return _grid_edges(math.isqrt(n), g)
    m = max(1, n * degree // 2)
    return _rmat_edges(n, m, g) if family == "rmat" else _er_edges(n, m, g)


def _csc(family, n, degree, g):
    """Undirected graph as int32 CSC on the GPU: sorted columns, no loops, no
    repeats."""
    u, v = _edges(family, n, degree, g)
    ok = u != v
    u, v = u[ok], v[ok]
    key = torch.unique(torch.cat([v * n + u, u * n + v]))
    del u, v
    col = torch.div(key, n, rounding_mode="floor")
    row = (key - col * n).to(torch.int32)
    cp = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    cp[1:] = torch.cumsum(torch.bincount(col, minlength=n), 0)
    return cp.to(torch.int32), row


def _entry_roots(cp, row, k, g):
    """k roots, each the source of a random entry: vertices by degree, so that
    a root lies in the giant component.  On a grid (degrees 0..6) the vertex
    is one of degree 4 at least."""
    deg = (cp[1:] - cp[:-1]).long()
    most = int(deg.max())
    if most <= 6:
        ok = torch.nonzero(deg >= min(4, most)).reshape(-1)
        return ok[torch.randint(ok.numel(), (k,), generator=g, device=DEV)].to(torch.int32)
    return row[torch.randint(row.numel(), (k,), generator=g, device=DEV)]


class _Graph:
    """A resident graph made from CSC arrays already on the device."""

    def __init__(self, cp, row, n):
        self.handle = ctypes.c_void_p()
        rc = tb.lib().tbfs_graph_create_csc(ctypes.cast(cp.data_ptr(), _I32P), ctypes.cast(row.data_ptr(), _I32P), n,
                                            row.numel(), SYMMETRIC | DEVICE_PTRS, ctypes.byref(self.handle))
        _ok(rc)
        self.n = n

    def __del__(self):
        if self.handle:
            tb.lib().tbfs_graph_destroy(self.handle)


def _ok(rc):
    if rc:
        raise RuntimeError(tb.lib().tbfs_last_error().decode())


def _device_options(sigma, mode="auto"):
    return tb.make_options(mode, sigma, outputs_on_device=True)


def _family_sizes(case):
    """(family, n) of the graphs of an arena or a server: sizes evenly spread
    over the logarithm, families in turn."""
    count, kinds = case["graphs"], ("rmat", "grid", "er")
    out = []
    for i in range(count):
        n = int(2.0 ** (case["lo"] + (case["hi"] - case["lo"]) * i / max(1, count - 1)))
        out.append((kinds[i % 3], math.isqrt(n) ** 2 if i % 3 == 1 else n))
    return out


# ----------------------------------------------------------------- states ---

def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind == "fresh":
        n, undirected = case["n"], case["undirected"]
        u, v = _edges(case["family"], n, case["degree"], g)
        u, v = u.to(torch.int32), v.to(torch.int32)
        root = int(u[int(torch.randint(u.numel(), (1,), generator=g, device=DEV))])
        return {"kind": kind, "n": n, "u": u, "v": v, "root": root, "opt": _device_options(case["sigma"]),
                "flags": DROP_LOOPS | DEDUP | (SYMMETRIZE if undirected else 0),
                "S": torch.empty(n, dtype=torch.int32, device=DEV),
                "sigma": torch.empty(n, dtype=torch.int64, device=DEV) if case["sigma"] else None}
    if kind == "arena":
        cps, rows, roots = [], [], []
        for family, n in _family_sizes(case):
            cp, row = _csc(family, n, 16, g)
            cps.append(cp)
            rows.append(row)
            roots.append(_entry_roots(cp, row, 1, g))
        n = np.array([cp.numel() - 1 for cp in cps], np.int32)
        nnz = np.array([row.numel() for row in rows], np.int64)
        cp, row = torch.cat(cps).cpu().numpy(), torch.cat(rows).cpu().numpy()
        h = ctypes.c_void_p()
        _ok(tb.lib().tbfs_arena_create(len(n), n.ctypes.data_as(_I32P), nnz.ctypes.data_as(_I64P), cp.ctypes.data_as(_I32P),
                                       row.ctypes.data_as(_I32P), SYMMETRIC, ctypes.byref(h)))
        total = int(n.sum())
        return {"kind": kind, "arena": _Arena(h), "roots": torch.cat(roots).cpu().numpy(), "opt": _device_options(case["sigma"], "td"),
                "S": torch.empty(total, dtype=torch.int32, device=DEV),
                "sigma": torch.empty(total, dtype=torch.int64, device=DEV) if case["sigma"] else None}
    if kind == "serve":
        graphs, roots = [], []
        for family, n in _family_sizes(case):
            cp, row = _csc(family, n, 16, g)
            graphs.append(_Graph(cp, row, n))
            roots.append(_entry_roots(cp, row, -(-case["queries"] // case["graphs"]), g).tolist())
        asked = [(graphs[i % len(graphs)], roots[i % len(graphs)][i // len(graphs)]) for i in range(case["queries"])]
        return {"kind": kind, "server": tb.Server(max_slots=64, mem_budget=1 << 30), "asked": asked, "sigma": case["sigma"]}
    n = case["n"]
    cp, row = _csc(case["family"], n, case["degree"], g)
    roots = _entry_roots(cp, row, case.get("k", 1), g).cpu().numpy()
    if kind == "dropin":
        entry = case["entry"]
        state = {"kind": kind, "entry": entry, "n": n, "nnz": row.numel(), "root": int(roots[0]), "I": row.cpu().numpy()}
        if entry == "cooc":
            col = torch.repeat_interleave(torch.arange(n, dtype=torch.int32, device=DEV), (cp[1:] - cp[:-1]).long())
            state["J"] = col.cpu().numpy()
        else:
            state["CP"] = cp.cpu().numpy()
            state["S"] = np.zeros(n, np.int32)
        if entry != "bu":
            state["sigma"] = np.zeros(n, np.int32 if entry == "tdbu" else np.float32)
        return state
    state = {"kind": kind, "graph": _Graph(cp, row, n), "roots": roots}
    if kind == "brandes":
        state["opt"] = _device_options(True)
        state["bc"] = torch.empty(n, dtype=torch.float64, device=DEV)
        return state
    state["opt"] = _device_options(case["sigma"], case.get("mode", "auto"))
    k = case.get("k", 1)
    shape = (n,) if kind == "bfs" else (k, n) if case["layout"] == ROOT_MAJOR else (n, k)
    state["layout"] = case.get("layout")
    state["S"] = torch.empty(shape, dtype=torch.int32, device=DEV)
    state["sigma"] = torch.empty(shape, dtype=torch.int64, device=DEV) if case["sigma"] else None
    return state


class _Arena:
    def __init__(self, handle):
        self.handle = handle

    def __del__(self):
        tb.lib().tbfs_arena_destroy(self.handle)


def _i32(t):
    return ctypes.cast(t.data_ptr(), _I32P)


def _i64(t):
    return ctypes.cast(t.data_ptr(), _I64P) if t is not None else None


def _pair(s):
    return [s["S"]] if s["sigma"] is None else [s["S"], s["sigma"]]


# ------------------------------------------------------------------- pass ---

def run(s):
    lib, kind = tb.lib(), s["kind"]
    if kind == "bfs":
        _ok(lib.tbfs_bfs(s["graph"].handle, int(s["roots"][0]), ctypes.byref(s["opt"]), _i32(s["S"]), _i64(s["sigma"]), None))
        return _pair(s)
    if kind == "fresh":
        h = ctypes.c_void_p()
        _ok(lib.tbfs_graph_create_edges(_i32(s["u"]), _i32(s["v"]), s["n"], s["u"].numel(), s["flags"], DEVICE_PTRS, ctypes.byref(h)))
        rc = lib.tbfs_bfs(h, s["root"], ctypes.byref(s["opt"]), _i32(s["S"]), _i64(s["sigma"]), None)
        lib.tbfs_graph_destroy(h)
        _ok(rc)
        return _pair(s)
    if kind == "batch":
        _ok(lib.tbfs_bfs_batch(s["graph"].handle, s["roots"].ctypes.data_as(_I32P), len(s["roots"]), ctypes.byref(s["opt"]),
                               s["layout"], s["S"].data_ptr(), s["sigma"].data_ptr() if s["sigma"] is not None else None, None))
        return _pair(s)
    if kind == "arena":
        _ok(lib.tbfs_arena_bfs(s["arena"].handle, s["roots"].ctypes.data_as(_I32P), ctypes.byref(s["opt"]), s["S"].data_ptr(),
                               s["sigma"].data_ptr() if s["sigma"] is not None else None, None))
        return _pair(s)
    if kind == "serve":
        server = s["server"]
        tickets = [server.submit(g, r, sigma=s["sigma"]) for g, r in s["asked"]]
        got = [server.wait(t)[0] for t in tickets]
        return [[r.S, r.sigma] if s["sigma"] else [r.S] for r in got]
    if kind == "dropin":
        return _dropin(s)
    _ok(lib.tbfs_brandes(s["graph"].handle, s["roots"].ctypes.data_as(_I32P), len(s["roots"]), ctypes.byref(s["opt"]),
                         s["bc"].data_ptr(), None))
    return [s["bc"]]


def _dropin(s):
    r, nz, n = s["root"], s["nnz"], s["n"]
    if s["entry"] == "td":
        _ok(tb.bfs_gpu_td_csc_sc(s["I"], s["CP"], s["S"], s["sigma"], r, nz, n, 1))
    elif s["entry"] == "bu":
        _ok(tb.bfs_gpu_bu_csc_sc(s["I"], s["CP"], s["S"], r, nz, n, 1, 1))
        return [s["S"]]
    elif s["entry"] == "tdbu":
        _ok(tb.bfs_gpu_tdbu_csc_sc(s["I"], s["CP"], s["S"], s["sigma"], r, nz, n, 1, 1))
    else:
        _ok(tb.bfs_gpu_td_cooc_sc(s["I"], s["J"], s["sigma"], r, nz, n, 1))
        return [s["sigma"]]
    return [s["S"], s["sigma"]]


# ------------------------------------------------------------------- work ---

def _entries(family, n, degree):
    """List entries of the undirected graph, about."""
    return 3.62 * n if family == "grid" else 0.95 * n * degree


def work(case):
    """Every list entry and list bound read once, every output written once
    (a fresh graph: also its edge list read and its lists written)."""
    kind = case["kind"]
    if kind in ("arena", "serve"):
        sizes = _family_sizes(case)
        times = 1.0 if kind == "arena" else case["queries"] / case["graphs"]
        per = 12 if case["sigma"] else 4
        return {"bytes": times * sum(4 * _entries(f, n, 16) + (4 + per) * n for f, n in sizes), "flops": 0}
    n = case["n"]
    nnz = _entries(case["family"], n, case["degree"])
    if kind == "dropin":
        lists = 8 * nnz if case["entry"] == "cooc" else 4 * nnz + 4 * n
        return {"bytes": lists + (4 if case["entry"] in ("bu", "cooc") else 8) * n, "flops": 0}
    if kind == "brandes":
        return {"bytes": 4 * nnz + 4 * n + 8 * n, "flops": 2 * nnz * case["k"]}
    out = (12 if case["sigma"] else 4) * n * case.get("k", 1)
    if kind == "fresh":
        m = n * case["degree"] // 2
        return {"bytes": 8 * m + (8 if case["undirected"] else 4) * nnz + 4 * n + out, "flops": 0}
    return {"bytes": 4 * nnz + 4 * n + out, "flops": 0}


# ------------------------------------------------------------------ exact ---

def _levels(cp, row, n, root):
    """Depths and path counts by whole-graph steps over all entries, and the
    entries that join a level to the next (sources, targets) per level."""
    col = torch.repeat_interleave(torch.arange(n, device=DEV), (cp[1:] - cp[:-1]).long())
    src = row.long()
    S = torch.full((n,), -1, dtype=torch.int32, device=DEV)
    sigma = torch.zeros(n, dtype=torch.int64, device=DEV)
    S[root], sigma[root] = 0, 1
    steps, d = [], 0
    while True:
        on = (S[src] == d) & (S[col] == -1)
        a, b = src[on], col[on]
        if not a.numel():
            return S, sigma, steps
        S[b] = d + 1
        sigma.index_add_(0, b, sigma[a])
        steps.append((a, b))
        d += 1


def exact(case, seed):
    """Single traversals and betweenness as plain torch gives them; the other
    kinds return whole numbers of many traversals and have none here."""
    if case["kind"] not in ("bfs", "brandes"):
        return None
    g = _gen(seed)
    n = case["n"]
    cp, row = _csc(case["family"], n, case["degree"], g)
    roots = _entry_roots(cp, row, case.get("k", 1), g).tolist()
    if case["kind"] == "bfs":
        S, sigma, _ = _levels(cp, row, n, roots[0])
        return [S, sigma] if case["sigma"] else [S]
    bc = torch.zeros(n, dtype=torch.float64, device=DEV)
    for root in roots:
        S, sigma, steps = _levels(cp, row, n, root)
        sg = sigma.double()
        delta = torch.zeros(n, dtype=torch.float64, device=DEV)
        for a, b in reversed(steps):
            delta.index_add_(0, a, sg[a] / sg[b] * (1 + delta[b]))
        delta[root] = 0
        bc += delta
    return [bc]
