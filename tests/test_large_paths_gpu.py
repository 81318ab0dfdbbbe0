"""GPU: the forms that only large graphs take, against the oracle or FP64.

WCC skips edges inside the largest sampled set by a bit per vertex (from
524,288 buckets), PageRank tells the runs of its segmented sums by position
(from 8,388,608 edges), and a member's triangle count sorts the oriented edges
by owner (from 524,288 directed edges)."""
import numpy as np
import pytest

import meerkat_b200 as mk
from helpers import make_pair, to_dev
from oracle import OracleGraph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("weighted", [False, True])
def test_wcc_with_a_set_that_holds_most_vertices(weighted):
    """A giant set, paths and single vertices beside it; then calls that
    reuse the words the bits were kept in: repairs after deletes inside and
    outside the giant set, an increment, and another static pass."""
    V, core = 600000, 500000
    rng = np.random.default_rng(5)
    ids = rng.permutation(V).astype(np.uint32)
    paths = ids[core:core + 80000].reshape(-1, 50)
    s = np.concatenate([ids[rng.integers(0, core, 1200000)], paths[:, :-1].ravel()])
    d = np.concatenate([ids[rng.integers(0, core, 1200000)], paths[:, 1:].ravel()])
    key = np.unique((s.astype(np.uint64) << 32 | d)[s != d])
    s, d = (key >> 32).astype(np.uint32), (key & 0xFFFFFFFF).astype(np.uint32)
    G, O = make_pair(V, s, d, np.ones(len(s), np.uint32), weighted=weighted, hints="ones")
    assert G.info()["num_buckets"] >= 1 << 19
    wcc = mk.WCC(G)
    for _ in range(2):
        wcc.Static()
        np.testing.assert_array_equal(wcc.Labels(), O.wcc())
    order = rng.permutation(len(s))
    for k, n in enumerate((40, 20000)):
        gone = order[k * 20000:k * 20000 + n]
        ds, dd = to_dev(s[gone]), to_dev(d[gone])
        G.DeleteEdges(ds, dd)
        O.delete(s[gone], d[gone])
        wcc.Decremental(ds, dd)
        np.testing.assert_array_equal(wcc.Labels(), O.wcc())
        bs, bd = rng.integers(0, V, 300).astype(np.uint32), rng.integers(0, V, 300).astype(np.uint32)
        ts, td = to_dev(bs), to_dev(bd)
        G.InsertEdges(ts, td, vals=to_dev(np.ones(300, np.uint32)) if weighted else None)
        O.insert(bs[bs != bd], bd[bs != bd])
        wcc.Incremental(ts, td)
        np.testing.assert_array_equal(wcc.Labels(), O.wcc())
        wcc.Static()
        np.testing.assert_array_equal(wcc.Labels(), O.wcc())


def test_pagerank_above_eight_million_edges():
    """Skewed in-degrees (hubs, rows inside and across the 32-edge steps,
    vertices without in- or out-edges) against FP64 power iteration."""
    V = 1 << 19
    s, d, _ = mk.gen_rmat(19, 12000000, seed=6)
    key = np.unique((s.astype(np.uint64) << 32 | d)[s != d])
    s, d = (key >> 32).astype(np.int64), (key & 0xFFFFFFFF).astype(np.int64)
    assert len(s) > 8 << 20
    G = mk.DynamicGraph(V, degree_hints=np.bincount(d, minlength=V).astype(np.uint32), reverse=True)
    G.InsertEdges(to_dev(s), to_dev(d))
    assert G.sync() == 0
    pr = mk.PageRank(G, 0.85, 1e-6, V, np.bincount(s, minlength=V).astype(np.uint32), 300)
    pr.Static()
    got = pr.Values().astype(np.float64)
    deg = np.bincount(s, minlength=V)
    damping = float(np.float32(0.85))  # the entry point takes a 32-bit number
    want, moved = np.full(V, 1.0 / V), 1.0
    while moved > 1e-13:
        nx = (1 - damping) / V + damping * (np.bincount(d, weights=want[s] / deg[s], minlength=V)
                                            + want[deg == 0].sum() / V)
        moved, want = np.abs(nx - want).sum(), nx
    assert np.abs(got - want).sum() <= 1e-6  # the solver's own stopping bound


@pytest.mark.parametrize("weighted", [False, True])
def test_tc_range_with_edges_sorted_by_owner(weighted):
    """The owner lists take the place of the member's CSR, row ids and degree
    counts; with reciprocal edges, a list longer than a warp takes (1,024
    entries: a clique of 1,100 vertices), and after deletes."""
    n, lead = 30000, 100
    rng = np.random.default_rng(9)
    a, b = np.triu_indices(1100, 1)
    s, d, _ = mk.gen_rmat(14, 400000, seed=2)
    s = np.concatenate([a, s, d[:90000], rng.integers(0, n, 200000)]).astype(np.uint32)
    d = np.concatenate([b, d, s[len(a):len(a) + 90000], rng.integers(0, n, 200000)]).astype(np.uint32)
    keep = s != d
    s, d = s[keep], d[keep]
    hints = [np.zeros(lead, np.uint32), np.bincount(s, minlength=n).astype(np.uint32), np.zeros(50, np.uint32)]
    gs = mk.GraphSet([lead, n, 50], degree_hints=hints, weighted=weighted)
    w = to_dev(np.ones(len(s), np.uint32)) if weighted else None
    gs.graph.InsertEdges(to_dev(s + lead), to_dev(d + lead), vals=w)
    assert gs.graph.sync() == 0 and gs.graph.count_edges(lead, lead + n) >= 1 << 19
    O = OracleGraph(n)
    O.insert(s, d)
    t = mk.TCRange(gs.graph)
    for _ in range(2):
        t.Run(lead, lead + n)
        assert t.GetCount() == O.triangles()
    gs.graph.DeleteEdges(to_dev(s[::9] + lead), to_dev(d[::9] + lead))
    O.delete(s[::9], d[::9])
    t.Run(lead, lead + n)
    assert t.GetCount() == O.triangles()
