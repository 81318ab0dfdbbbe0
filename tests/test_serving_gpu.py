"""Serving loop: every query answer is the same when the request is served
in a coalesced round with other graphs' requests and when it is served alone,
and equals the oracle's answer on its graph after the updates that arrived
before it."""
import copy

import numpy as np
import pytest

import meerkat_b200 as mk
from meerkat_b200 import serving as S
from oracle import OracleGraph

PR_L1_TOL = 1e-6


def make_server(seed):
    nv, ne = S.make_graph_sizes(6, 8, 11, 8, seed)
    gs, edges = S.build_set(nv, ne, seed)
    wl = S.Workload(nv, ne, seed)
    return gs, edges, wl


def oracle_answers(nv, edges_h, voff, reqs, pool):
    """Replays every graph's requests in arrival order on the oracle."""
    src, dst, w = edges_h
    Os = []
    for g in range(len(nv)):
        Os.append(OracleGraph(int(nv[g])))
    # initial edges of each member (R-MAT, duplicates collapse in the oracle)
    owner = np.searchsorted(voff, src, side="right") - 1
    for g in range(len(nv)):
        m = owner == g
        Os[g].insert((src[m] - voff[g]).astype(np.uint32), (dst[m] - voff[g]).astype(np.uint32),
                     w[m])
    ps, pd, pw = pool
    out = {}
    for r in sorted(reqs, key=lambda r: r.arrival):
        O, base = Os[r.graph], int(voff[r.graph])
        if r.kind == S.INSERT:
            O.insert((ps[r.lo:r.hi] - base).astype(np.uint32), (pd[r.lo:r.hi] - base).astype(np.uint32),
                     pw[r.lo:r.hi])
        elif r.kind == S.DELETE:
            O.delete((ps[r.lo:r.hi] - base).astype(np.uint32), (pd[r.lo:r.hi] - base).astype(np.uint32))
        elif r.kind == S.BFS_Q:
            out[r.rid] = O.bfs(r.source)
        elif r.kind == S.SSSP_Q:
            out[r.rid] = O.sssp(r.source)
        elif r.kind == S.WCC_Q:
            out[r.rid] = O.wcc()
        elif r.kind == S.TC_Q:
            out[r.rid] = O.triangles()
        elif r.kind == S.PAGERANK_Q:
            out[r.rid] = O.pagerank(0.85, 1e-14)[0]
    return out


def h(t):
    return t.cpu().numpy().view(np.uint32).astype(np.int64)


@pytest.mark.gpu
def test_alone_and_coalesced_answers_match_each_other_and_the_oracle():
    seed = 21
    gsA, edgesA, wlA = make_server(seed)
    gsB, edgesB, wlB = make_server(seed)
    # the same seeded log on both sets; every request arrives at once, so the
    # coalesced server packs up to one request per graph into each round
    reqsA = S.make_requests(wlA, edgesA, 90, rate=1e7, seed=seed + 1, upd_lo=10, upd_hi=3000)
    reqsB = S.make_requests(wlB, edgesB, 90, rate=1e7, seed=seed + 1, upd_lo=10, upd_hi=3000)
    import torch
    assert torch.equal(wlA.pool_src, wlB.pool_src) and torch.equal(wlA.pool_dst, wlB.pool_dst)
    kinds = {r.kind for r in reqsA}
    assert kinds == set(range(7)), kinds
    voff = gsA.offsets.astype(np.int64)
    oracle = oracle_answers(wlA.num_vertices, tuple(h(x) for x in edgesA), voff, reqsA,
                            (h(wlA.pool_src), h(wlA.pool_dst), h(wlA.pool_w)))
    A = S.GraphServer(gsA, budget_bytes=1 << 36, record=True)
    B = S.GraphServer(gsB, budget_bytes=1 << 36, record=True)
    ra = A.run(reqsA, wlA, mode="coalesced")
    rb = B.run(reqsB, wlB, mode="alone")
    assert rb["rounds"] == len(reqsB) and ra["rounds"] < len(reqsA)
    for x, y in zip(reqsA, reqsB):
        assert x.rid == y.rid and x.kind == y.kind
        if x.kind in (S.INSERT, S.DELETE):
            continue
        want = oracle[x.rid]
        if x.kind == S.PAGERANK_Q:
            assert np.abs(x.result.astype(np.float64) - want).sum() <= PR_L1_TOL
            assert np.abs(y.result.astype(np.float64) - want).sum() <= PR_L1_TOL
            assert np.abs(x.result.astype(np.float64) - y.result).sum() <= PR_L1_TOL
        elif x.kind == S.TC_Q:
            assert x.result == y.result == want
        else:
            np.testing.assert_array_equal(x.result, want)
            np.testing.assert_array_equal(y.result, want)
    A.close()
    B.close()


@pytest.mark.gpu
def test_inserts_beyond_the_slab_pool_are_refused_not_failed():
    """Admission by slab-pool headroom: with the pool's capacity lowered on
    the host, large inserts are refused at admission (status "rejected")
    instead of running out of slabs on the device; everything else is
    served and the graph stays consistent."""
    seed = 5
    gs, edges, wl = make_server(seed)
    reqs = S.make_requests(wl, edges, 40, rate=1e7, seed=7,
                           mix=(0.5, 0.1, 0.2, 0, 0, 0.2, 0), upd_lo=100, upd_hi=3000)
    srv = S.GraphServer(gs, budget_bytes=1 << 40)
    srv.pool_cap = srv.slabs_used + 1024 + 500  # room for one small insert at most
    out = srv.run(reqs, wl, mode="coalesced")
    rej = [r for r in reqs if r.status != "ok"]
    assert rej and all(r.kind == S.INSERT and r.hi - r.lo > 500 for r in rej)
    assert out["rejected"] == len(rej)
    assert all(r.done >= 0 for r in reqs)
    assert gs.graph.sync() == 0
    srv.close()


@pytest.mark.gpu
@pytest.mark.parametrize("roomy", [True, False])
def test_pagerank_scratch_stays_within_what_the_server_accounts_for(roomy):
    """PageRank requests allocate nothing once the server stands, on the
    member with the most vertices and on one that has grown past the scratch
    (then pushed from the slabs), and their answers stay the oracle's."""
    import torch
    gs, edges, wl = make_server(17)
    nv, voff = wl.num_vertices, gs.offsets.astype(np.int64)
    budget = 1 << 40
    if not roomy:  # what stands and the largest triangle count's scratch, no more
        twin = make_server(17)[0]
        probe = S.GraphServer(twin, budget_bytes=budget, max_update=1000)
        tc = max(S.TC_BYTES_PER_EDGE * twin.graph.count_edges(voff[m], voff[m + 1])
                 + S.TC_BYTES_PER_VERTEX * int(nv[m]) for m in range(len(nv)))
        budget = probe.resident - 8 * probe.pagerank_edges + tc + 8 * 1024
        probe.close()
    srv = S.GraphServer(gs, budget_bytes=budget, record=True, max_update=1000)
    assert srv.resident <= budget
    assert srv.pagerank_edges >= wl.num_edges.max() if roomy else srv.pagerank_edges == 1024
    g = int(np.argmax(nv))
    Os = OracleGraph(int(nv[g]))
    own = (h(edges[0]) >= voff[g]) & (h(edges[0]) < voff[g + 1])
    Os.insert((h(edges[0])[own] - voff[g]).astype(np.uint32), (h(edges[1])[own] - voff[g]).astype(np.uint32))
    rng = np.random.default_rng(3)
    for grow in (0, 40000):
        if grow:
            u = rng.integers(0, nv[g], grow)
            v = (u + 1 + rng.integers(0, nv[g] - 1, grow)) % nv[g]
            td = lambda a: torch.from_numpy(a.astype(np.int32)).cuda()  # noqa: E731
            gs.graph.InsertEdges(td(u + voff[g]), td(v + voff[g]), vals=td(np.ones(grow)))
            Os.insert(u.astype(np.uint32), v.astype(np.uint32))
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        r = S.Request(rid=0, graph=g, kind=S.PAGERANK_Q, arrival=0.0)
        srv.run_heavy(r, srv.heavy)
        torch.cuda.synchronize()
        assert torch.cuda.mem_get_info()[0] == free
        assert r.status == "ok"
        assert np.abs(r.result.astype(np.float64) - Os.pagerank(0.85, 1e-14)[0]).sum() <= PR_L1_TOL
    srv.close()


@pytest.mark.gpu
def test_triangle_counts_beyond_the_budget_are_refused():
    seed = 6
    gs, edges, wl = make_server(seed)
    reqs = S.make_requests(wl, edges, 20, rate=1e7, seed=9, mix=(0, 0, 0, 0, 0, 1, 0))
    srv = S.GraphServer(gs, budget_bytes=1 << 40)
    srv.budget = srv.resident  # no room for any scratch beyond what is held
    srv.tc_bytes = 0
    out = srv.run(reqs, wl, mode="coalesced")
    assert out["rejected"] == len(reqs)
    assert all(r.status == "rejected" for r in reqs)
    srv.close()


@pytest.mark.gpu
def test_saturated_coalesced_run_overlaps_heavy_and_fast_work():
    """All requests at once: the coalesced server answers every request and
    finishes no later than the one-at-a-time sequence of the same log."""
    seed = 8
    gsA, edgesA, wlA = make_server(seed)
    reqs = S.make_requests(wlA, edgesA, 80, rate=1e9, seed=seed + 1, upd_lo=10, upd_hi=3000)
    srv = S.GraphServer(gsA, budget_bytes=1 << 40)
    srv.run([S.Request(r.rid, r.graph, r.kind, r.arrival, r.source, r.lo, r.hi) for r in reqs[:8]],
            wlA, mode="coalesced")  # warm-up
    a = srv.run([S.Request(r.rid, r.graph, r.kind, r.arrival, r.source, r.lo, r.hi) for r in reqs],
                wlA, mode="coalesced")
    b = srv.run([S.Request(r.rid, r.graph, r.kind, r.arrival, r.source, r.lo, r.hi) for r in reqs],
                wlA, mode="alone")
    assert a["rejected"] == b["rejected"] == 0
    assert a["rounds"] < b["rounds"] == len(reqs)
    assert a["throughput_rps"] > 0.9 * b["throughput_rps"]
    srv.close()


def test_request_log_is_seeded():
    nv, ne = S.make_graph_sizes(8, 10, 14, 16, 3)
    nv2, ne2 = S.make_graph_sizes(8, 10, 14, 16, 3)
    assert (nv == nv2).all() and (ne == 16 * nv).all()
    assert nv.min() >= 1 << 10 and nv.max() <= 1 << 14
