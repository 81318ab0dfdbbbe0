"""Workloads of the framework as a user's program runs them, for timing.

Every case is a dict of plain values.  `prepare` makes what a program holds
before the call (graphs on the GPU, algorithm handles, update batches) from a
seed alone, `run` is one pass through the public entry points and `work` the
bytes one pass cannot do without.  Graphs are R-MAT (a, b, c, d = 0.57, 0.19,
0.19, 0.05), whose vertex count need not be a power of two, or a 4-neighbour
grid with 1 % long-range shortcuts.

Results are read where a GPU program reads them: the packed distances, labels
and ranks in device memory.  Parents are left out of the outputs, since any
shortest-path tree is a right answer; distances, labels, degrees and counts
are unique.

Updates change the graph, so the dynamic cases cycle through a ring of
disjoint batches: pass k deletes batch k and inserts batch k - 1 again, as in
the mixed update batches of the benchmark.  Deleted slots are never reused,
so these graphs are built with room to grow (`slack` times the degree hints),
as a program with lasting churn builds them.
"""
import ctypes
import math

import numpy as np
import torch

import meerkat_b200 as mk

DEV = "cuda:0"
CUT_S, CUT_D0, CUT_D1 = 0.76, 0.57, 0.95  # quadrant a | b | c | d of one R-MAT level


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _rmat_ids(g, n, bits):
    """n R-MAT id pairs of `bits` bits each."""
    s = torch.zeros(n, dtype=torch.int64, device=DEV)
    d = torch.zeros(n, dtype=torch.int64, device=DEV)
    for _ in range(bits):
        r = torch.rand(n, generator=g, device=DEV)
        s.mul_(2).add_(r >= CUT_S)
        d.mul_(2).add_(((r >= CUT_D0) & (r < CUT_S)) | (r >= CUT_D1))
    return s, d


def _rmat(g, vertices, edges):
    """Distinct directed R-MAT edges without self-loops, in random order."""
    bits = max(1, (vertices - 1).bit_length())
    s, d = _rmat_ids(g, edges, bits)
    s, d = s * vertices >> bits, d * vertices >> bits
    key = torch.unique((s * vertices + d)[s != d])
    key = key[torch.randperm(key.numel(), generator=g, device=DEV)]
    return (key // vertices).to(torch.int32), (key % vertices).to(torch.int32)


def _grid(g, side):
    """Both directions of a side x side grid, plus 1 % random shortcuts."""
    v = torch.arange(side * side, device=DEV)
    right, down = v[v % side < side - 1], v[: side * (side - 1)]
    far = torch.randint(side * side, (2, 4 * side * side // 100), generator=g, device=DEV)
    s = torch.cat([right, right + 1, down, down + side, far[0]])
    d = torch.cat([right + 1, right, down + side, down, far[1]])
    key = torch.unique((s * (side * side) + d)[s != d])
    key = key[torch.randperm(key.numel(), generator=g, device=DEV)]
    return (key // (side * side)).to(torch.int32), (key % (side * side)).to(torch.int32)


def _weights(g, n, most):
    return torch.randint(1, most + 1, (n,), generator=g, device=DEV, dtype=torch.int32)


def _hints(ids, vertices, slack=1):
    return (torch.bincount(ids, minlength=vertices) * slack).to(torch.int32).cpu().numpy().view(np.uint32)


def _edges(case, g):
    if case.get("grid"):
        return _grid(g, case["grid"])
    return _rmat(g, case["vertices"], case["edges"])


def _vertices(case):
    return case["grid"] ** 2 if case.get("grid") else case["vertices"]


# --------------------------------------------------------------------------
# results in device memory
# --------------------------------------------------------------------------
class _Device:
    """A device array of the framework, as torch takes it over.  `owner` is
    the object that holds the memory: it lives as long as the tensor."""

    def __init__(self, owner, ptr, shape, typestr, strides):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr,
                                         "strides": strides, "version": 2}


def _tensor(owner, ptr, shape, typestr="<i4", strides=None):
    return torch.as_tensor(_Device(owner, ptr, shape, typestr, strides), device=DEV)


def _distances(algo, owner=None):
    """The distance words of the packed dist << 32 | parent array."""
    return _tensor(owner or algo, algo.packed_ptr() + 4, (algo.G.num_vertices,), strides=(8,))


def _labels(wcc, owner=None):
    p = ctypes.c_void_p()
    mk.lib().mk_wcc_labels_device(wcc._h, ctypes.byref(p))
    return _tensor(owner or wcc, p.value, (wcc.G.num_vertices,))


def _ranks(pr):
    p = ctypes.c_void_p()
    mk.lib().mk_pagerank_values_device(pr._h, ctypes.byref(p))
    return _tensor(pr, p.value, (pr.G.num_vertices,), "<f4")


# --------------------------------------------------------------------------
# lookups: membership of a batch of pairs, half of them present
# --------------------------------------------------------------------------
def _prepare_search(case, seed):
    g = _gen(seed)
    V = case["vertices"]
    s, d = _rmat(g, V, case["edges"])
    G = mk.DynamicGraph(V, degree_hints=_hints(s, V), weighted=case["weighted"])
    G.InsertEdges(s, d, vals=_weights(g, s.numel(), 1000) if case["weighted"] else None)
    n = case["queries"]
    at = torch.randint(s.numel(), (n,), generator=g, device=DEV)
    qs, qd = s[at], d[at]
    other = torch.randint(V, (n,), generator=g, device=DEV, dtype=torch.int32)
    qd = torch.where(torch.rand(n, generator=g, device=DEV) < 0.5, qd, other)
    found = torch.empty(n, dtype=torch.uint8, device=DEV)
    w = torch.empty(n, dtype=torch.int32, device=DEV) if case["weighted"] else None
    return {"G": G, "q": (qs, qd, found, w)}


def _run_search(st):
    s, d, found, w = st["q"]
    st["G"].SearchEdges(s, d, found, weights=w)
    return (found, w) if w is not None else found


def _work_search(case):
    # pair in, one slab line probed, flag (and weight) out
    return case["queries"] * (8 + 128 + 1 + (4 if case["weighted"] else 0))


# --------------------------------------------------------------------------
# refresh: a feed that reports edges again and again.  The batch's edges are
# in the graph already, the smaller weight stays, and the feed reads back what
# the graph now holds
# --------------------------------------------------------------------------
def _prepare_refresh(case, seed):
    g = _gen(seed)
    V = case["vertices"]
    s, d = _rmat(g, V, case["edges"])
    G = mk.DynamicGraph(V, degree_hints=_hints(s, V), weighted=True)
    G.InsertEdges(s, d, vals=_weights(g, s.numel(), 1000))
    n = case["batch"]
    at = torch.randint(s.numel(), (n,), generator=g, device=DEV)
    G.reserve_batch(n)
    return {"G": G, "batch": (s[at], d[at]), "w": _weights(g, n, 1000),
            "found": torch.empty(n, dtype=torch.uint8, device=DEV),
            "now": torch.empty(n, dtype=torch.int32, device=DEV)}


def _run_refresh(st):
    s, d = st["batch"]
    st["G"].InsertEdges(s, d, vals=st["w"])
    st["G"].SearchEdges(s, d, st["found"], weights=st["now"])
    return st["found"], st["now"]


def _work_refresh(case):
    # pair and weight in and a slab line probed by the update, pair and line
    # again by the read back; flag and weight out
    return case["batch"] * (12 + 128 + 8 + 128 + 5)


# --------------------------------------------------------------------------
# static algorithms on one graph
# --------------------------------------------------------------------------
def _prepare_static(case, seed):
    g = _gen(seed)
    V, algo = _vertices(case), case["algo"]
    s, d = _edges(case, g)
    if algo == "tc":  # symmetric graph
        key = torch.unique(torch.cat([s.long() * V + d, d.long() * V + s]))
        s, d = (key // V).to(torch.int32), (key % V).to(torch.int32)
    if algo == "pagerank":
        G = mk.DynamicGraph(V, degree_hints=_hints(d, V), reverse=True)
        G.InsertEdges(s, d)
        pr = mk.PageRank(G, 0.85, 1e-6, out_degree=_hints(s, V))
        return {"G": G, "algo": pr, "kind": algo}
    w = _weights(g, s.numel(), 1000) if case["weighted"] else None
    G = mk.DynamicGraph(V, degree_hints=_hints(s, V), weighted=case["weighted"])
    G.InsertEdges(s, d, vals=w)
    st = {"G": G, "kind": algo}
    source = int(s[0]) if not case.get("grid") else (V + case["grid"]) // 2
    if algo in ("bfs", "sssp"):
        st["algo"] = (mk.BFS if algo == "bfs" else mk.SSSP)(G, source)
        st["out"] = _distances(st["algo"])
    elif algo == "wcc":
        st["algo"] = mk.WCC(G)
        st["out"] = _labels(st["algo"])
    else:
        st["algo"] = mk.TC(G)
    return st


def _run_static(st):
    a = st["algo"]
    a.Static(timed=False)
    if st["kind"] == "pagerank":
        return _ranks(a)
    if st["kind"] == "tc":
        return a.GetCount()
    return st["out"]


def _work_static(case):
    V = _vertices(case)
    E = 4 * V if case.get("grid") else case["edges"]
    return {"bfs": 4 * E + 16 * V,        # every edge's key once, offsets and the result per vertex
            "sssp": 8 * E + 16 * V,       # keys and weights
            "wcc": 4 * E + 12 * V,
            "pagerank": 8 * E + 16 * V,   # one sweep: keys and contributions
            "tc": 8 * E + 8 * V}[case["algo"]]  # both directions of every edge once


# --------------------------------------------------------------------------
# streams: mixed update batches with the algorithms kept up to date
# --------------------------------------------------------------------------
def _prepare_stream(case, seed):
    g = _gen(seed)
    V, algos = _vertices(case), case["algos"].split("+")
    s, d = _edges(case, g)
    w = _weights(g, s.numel(), 1000) if case["weighted"] else None
    B = case["batch"]
    K = max(2, min(64, s.numel() // (2 * B)))
    ring = [(s[i * B:(i + 1) * B].clone(), d[i * B:(i + 1) * B].clone(),
             w[i * B:(i + 1) * B].clone() if w is not None else None) for i in range(K)]
    st = {"ring": ring, "k": 0, "algos": []}
    G = mk.DynamicGraph(V, degree_hints=_hints(s, V, case["slack"]), weighted=case["weighted"])
    graphs = [G]
    if case["reverse"]:
        graphs.append(mk.DynamicGraph(V, degree_hints=_hints(d, V, case["slack"]), weighted=case["weighted"],
                                      reverse=True))
    # the last batch of the ring is out of the graph when the stream starts
    keep = torch.ones(s.numel(), dtype=torch.bool, device=DEV)
    keep[(K - 1) * B:K * B] = False
    for H in graphs:
        H.InsertEdges(s[keep], d[keep], vals=w[keep] if w is not None else None)
        H.reserve_batch(B)
    torch.cuda.synchronize()
    source = int(torch.mode(s[:4096]).values) if not case.get("grid") else (V + case["grid"]) // 2
    out = []
    for name in algos:
        if name == "wcc":
            a = mk.WCC(G)
        else:
            a = (mk.BFS if name == "bfs" else mk.SSSP)(G, source)
        if case["reverse"]:
            a.set_reverse(graphs[1])
        a.Static()
        st["algos"].append(a)
        out.append(_labels(a) if name == "wcc" else _distances(a))
    st["graphs"], st["out"] = graphs, out
    return st


def _run_stream(st):
    ring, k = st["ring"], st["k"]
    gone, back = ring[k % len(ring)], ring[(k - 1) % len(ring)]
    for H in st["graphs"]:
        H.DeleteEdges(gone[0], gone[1])
    for a in st["algos"]:
        a.Decremental(gone[0], gone[1], timed=False)
    for H in st["graphs"]:
        H.InsertEdges(back[0], back[1], vals=back[2])
    for a in st["algos"]:
        a.Incremental(back[0], back[1], timed=False)
    st["k"] = k + 1
    return st["out"]


def _work_stream(case):
    # a slab line read and written per update (and graph); per algorithm the
    # batch's pairs and both ends' words
    graphs, algos = 2 if case["reverse"] else 1, len(case["algos"].split("+"))
    return 2 * case["batch"] * (graphs * (12 + 256) + algos * (8 + 16))


# --------------------------------------------------------------------------
# many small graphs: one update batch and one query per member and step
# --------------------------------------------------------------------------
def _members(case):
    """Vertex and edge counts of the members: the same for every seed."""
    r = np.random.default_rng(case["members"])
    n = case["members"]
    nv = np.exp(r.uniform(math.log(case["v_lo"]), math.log(case["v_hi"]), n)).astype(np.int64)
    deg = 1.0 / (1 / 4 - r.random(n) * (1 / 4 - 1 / 32))  # power law, exponent 2, on [4, 32]
    ne = np.maximum(64, np.round(nv * deg)).astype(np.int64)
    return nv, ne


def _set_edges(g, nv, ne):
    """Distinct R-MAT edges of every member (global ids), grouped by member
    and in random order inside it, and the members' edge counts."""
    off = np.concatenate([[0], np.cumsum(nv)])
    m = torch.repeat_interleave(torch.arange(len(nv), device=DEV), torch.from_numpy(ne).to(DEV))
    v, o = torch.from_numpy(nv).to(DEV)[m], torch.from_numpy(off[:-1]).to(DEV)[m]
    bits = 16
    s, d = _rmat_ids(g, m.numel(), bits)
    s, d = (s * v >> bits) + o, (d * v >> bits) + o
    key = torch.unique((s * int(off[-1]) + d)[s != d])
    key = key[torch.randperm(key.numel(), generator=g, device=DEV)]
    s, d = key // int(off[-1]), key % int(off[-1])
    m = torch.bucketize(s, torch.from_numpy(off[1:]).to(DEV), right=True)
    order = torch.argsort(m, stable=True)
    return off, s[order].to(torch.int32), d[order].to(torch.int32), m[order]


def _prepare_set(case, seed):
    g = _gen(seed)
    nv, ne = _members(case)
    off, s, d, m = _set_edges(g, nv, ne)
    n, V = len(nv), int(off[-1])
    w = _weights(g, s.numel(), 64) if case["weighted"] else None
    hints = _hints(s, V, case["slack"])
    gs = mk.GraphSet(nv, degree_hints=[hints[off[i]:off[i + 1]] for i in range(n)], weighted=case["weighted"])
    # ring of batches: a share of every member's edges each (U[0.5, 5] % of
    # the member, at least one)
    K = 10
    cnt = torch.bincount(m, minlength=n)
    first = torch.cumsum(cnt, 0) - cnt
    share = 0.005 + 0.045 * torch.rand(n, generator=g, device=DEV)
    take = (cnt * share).long().clamp(min=1)
    slot = (torch.arange(s.numel(), device=DEV) - first[m]) // take[m]
    ring = []
    for k in range(K):
        at = slot == k
        ring.append((s[at], d[at], w[at] if w is not None else None))
    keep = slot != K - 1
    gs.graph.InsertEdges(s[keep], d[keep], vals=w[keep] if w is not None else None)
    gs.graph.reserve_batch(max(b[0].numel() for b in ring))
    # breadth-first searches on the first half of the members, components on
    # the second; a search starts at an end of one of the member's edges
    query = (np.arange(n) >= n // 2).astype(np.uint8)
    src = s[first.clamp(max=s.numel() - 1)].cpu().numpy().astype(np.int64) - off[:-1]
    src = np.where((src >= 0) & (src < nv), src, 0).astype(np.uint32)
    r = mk.SetRunner(gs, query, src)
    mid = int(off[n // 2])
    torch.cuda.synchronize()
    return {"gs": gs, "runner": r, "ring": ring, "k": 0,
            "out": [_distances(r.bfs, r)[:mid], _labels(r.wcc, r)[mid:]]}


def _run_set(st):
    ring, k = st["ring"], st["k"]
    gone, back = ring[k % len(ring)], ring[(k - 1) % len(ring)]
    st["runner"].step(gone[0], gone[1], back[0], back[1], back[2])
    st["k"] = k + 1
    return st["out"]


def _work_set(case):
    _, ne = _members(case)
    nv = np.exp((math.log(case["v_lo"]) + math.log(case["v_hi"])) / 2) * case["members"]
    # every member's keys once, a word per vertex out, and the updates
    return int(4 * ne.sum() + 16 * nv + 2 * 0.0275 * ne.sum() * (8 + 256))


# --------------------------------------------------------------------------
# requests on one member of a resident set, as the serving loop runs them
# --------------------------------------------------------------------------
def _prepare_member(case, seed):
    g = _gen(seed)
    V = case["vertices"]
    sets = [_rmat(g, V, case["edges"]), _rmat(g, max(1024, V // 4), case["edges"] // 4)]
    nv = [V, max(1024, V // 4)]
    s = torch.cat([sets[0][0], sets[1][0] + V])
    d = torch.cat([sets[0][1], sets[1][1] + V])
    h = _hints(s, sum(nv))
    gs = mk.GraphSet(nv, degree_hints=[h[:V], h[V:]], weighted=case["weighted"])
    gs.graph.InsertEdges(s, d, vals=_weights(g, s.numel(), 1000) if case["weighted"] else None)
    st = {"gs": gs, "range": (0, V), "kind": case["request"]}
    if case["request"] == "pagerank":
        st["algo"] = mk.PageRankRange(gs.graph, V)
    else:
        st["algo"] = mk.TCRange(gs.graph)
        st["algo"].Run(0, V)
    torch.cuda.synchronize()
    return st


def _run_member(st):
    st["algo"].Run(*st["range"], timed=False)
    return st["algo"].Values() if st["kind"] == "pagerank" else st["algo"].GetCount()


def _work_member(case):
    # one sweep over the member's keys; ranks out, or both directions once
    return 8 * case["edges"] + 16 * case["vertices"]


# --------------------------------------------------------------------------
KINDS = {"search": (_prepare_search, _run_search, _work_search),
         "refresh": (_prepare_refresh, _run_refresh, _work_refresh),
         "static": (_prepare_static, _run_static, _work_static),
         "stream": (_prepare_stream, _run_stream, _work_stream),
         "set": (_prepare_set, _run_set, _work_set),
         "member": (_prepare_member, _run_member, _work_member)}


def listed():
    return [
        # the smallest call: a batch of lookups in a small graph
        {"name": "search-60k", "kind": "search", "vertices": 65536, "edges": 1048576, "weighted": False,
         "queries": 60013},
        # a large batch of edges reported again, weights upserted and read back
        {"name": "refresh-1M", "kind": "refresh", "vertices": 1048576, "edges": 16777216, "batch": 1000000},
        # the small benchmark graph under mixed batches of 10,000, one graph
        # kept, shortest paths and levels from one source kept up to date
        {"name": "stream-10k", "kind": "stream", "vertices": 65536, "edges": 1048576, "weighted": True, "batch": 5000,
         "algos": "bfs+sssp", "reverse": False, "slack": 4},
        # the large benchmark's mixed batches at a quarter of its size, with
        # the reverse copy that the repairs use: shortest paths and components
        {"name": "stream-500k", "kind": "stream", "vertices": 1048576, "edges": 16777216, "weighted": True,
         "batch": 250000, "algos": "sssp+wcc", "reverse": True, "slack": 4},
        # static recomputes on the large benchmark graph and on others of its
        # family: levels, shortest paths, components, ranks, triangles
        {"name": "bfs-67M", "kind": "static", "algo": "bfs", "vertices": 4194304, "edges": 67108864,
         "weighted": False},
        {"name": "sssp-16M", "kind": "static", "algo": "sssp", "vertices": 1048576, "edges": 16777216,
         "weighted": True},
        # a high-diameter graph: many small frontiers
        {"name": "sssp-grid", "kind": "static", "algo": "sssp", "grid": 1500, "weighted": True},
        {"name": "wcc-48M", "kind": "static", "algo": "wcc", "vertices": 3000001, "edges": 48000000,
         "weighted": False},
        {"name": "pagerank-32M", "kind": "static", "algo": "pagerank", "vertices": 2097152, "edges": 33554432,
         "weighted": False},
        {"name": "tc-8M", "kind": "static", "algo": "tc", "vertices": 524288, "edges": 8388608, "weighted": False},
        # many small graphs advanced together
        {"name": "set-512", "kind": "set", "members": 512, "v_lo": 1024, "v_hi": 65536, "weighted": False,
         "slack": 3},
        # the heavy request of the serving loop: ranks of one resident member
        {"name": "member-pagerank", "kind": "member", "request": "pagerank", "vertices": 262144, "edges": 4194304,
         "weighted": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["search", "refresh", "static", "static", "static", "static", "stream", "stream", "set", "member"])
    V = _log(rng, 20000, 3000000)
    E = int(min(48000000, V * rng.uniform(6, 20)))
    weighted = rng.random() < 0.5
    if kind == "search":
        return {"kind": kind, "vertices": V, "edges": E, "weighted": weighted, "queries": _log(rng, 1000, 4000000)}
    if kind == "refresh":
        return {"kind": kind, "vertices": V, "edges": E, "batch": _log(rng, 2000, 2000000)}
    if kind == "static":
        algo = rng.choice(["bfs", "sssp", "wcc", "pagerank", "tc"])
        if algo in ("sssp", "tc"):
            V = min(V, 1048576 if algo == "sssp" else 400000)
            E = int(V * rng.uniform(6, 16))
        if algo in ("bfs", "sssp", "wcc") and rng.random() < 0.25:
            return {"kind": kind, "algo": algo, "grid": _log(rng, 200, 1400), "weighted": algo == "sssp" or weighted}
        return {"kind": kind, "algo": algo, "vertices": V, "edges": E,
                "weighted": algo == "sssp" or (weighted and algo in ("bfs", "wcc"))}
    if kind == "stream":
        V = min(V, 1000000)
        E = int(V * rng.uniform(8, 16))
        algos = rng.choice(["bfs", "sssp", "wcc", "bfs+sssp", "bfs+wcc", "sssp+wcc"])
        return {"kind": kind, "vertices": V, "edges": E, "weighted": "sssp" in algos or weighted,
                "batch": max(500, int(E * rng.uniform(0.003, 0.02))), "algos": algos,
                "reverse": "bfs" not in algos and rng.random() < 0.7, "slack": 4}
    if kind == "set":
        lo = _log(rng, 1000, 8000)
        return {"kind": kind, "members": _log(rng, 100, 500), "v_lo": lo, "v_hi": _log(rng, lo + 1000, 65000),
                "weighted": weighted, "slack": 3}
    V = _log(rng, 20000, 262144)
    return {"kind": kind, "request": rng.choice(["pagerank", "tc"]), "vertices": V,
            "edges": int(V * rng.uniform(6, 16)), "weighted": weighted}


def prepare(case, seed):
    st = KINDS[case["kind"]][0](case, seed)
    st["run"] = KINDS[case["kind"]][1]
    return st


def run(state):
    return state["run"](state)


def work(case):
    return {"bytes": KINDS[case["kind"]][2](case), "flops": 0}


def _power_iteration(s, d, V, damping):
    """Ranks in 64 bits, iterated until they no longer move."""
    outdeg = torch.bincount(s, minlength=V).double()
    order = torch.argsort(d)
    s, d = s[order].long(), d[order].long()
    p = torch.full((V,), 1.0 / V, dtype=torch.float64, device=DEV)
    for _ in range(300):
        c = torch.where(outdeg > 0, p / outdeg.clamp(min=1), torch.zeros_like(p))
        q = torch.zeros_like(p).index_add_(0, d, c[s])
        q = (1 - damping) / V + damping * (q + p[outdeg == 0].sum() / V)
        moved = float((q - p).abs().sum())
        p = q
        if moved < 1e-13:
            break
    return p


def exact(case, seed):
    """The ranks in 64 bits; every other output is whole numbers."""
    g = _gen(seed)
    if case["kind"] == "static" and case["algo"] == "pagerank":
        s, d = _edges(case, g)
    elif case["kind"] == "member" and case["request"] == "pagerank":
        s, d = _rmat(g, case["vertices"], case["edges"])
    else:
        return None
    return _power_iteration(s, d, case["vertices"], 0.85)
