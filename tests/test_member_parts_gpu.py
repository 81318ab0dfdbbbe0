"""GPU: components of graph-set members that several CTAs share.

A member with more buckets than an SM's share is cut into 2, 4 or 8 parts,
whose sets are joined in a tournament.  One bucket per vertex here, so the
sizes stand on the edges of the rule (4,096 buckets a part) and of the 16-bit
local ids; shapes with one set, with many, and with long chains."""
import numpy as np
import pytest

import meerkat_b200 as mk
from helpers import to_dev
from oracle import OracleGraph

pytestmark = pytest.mark.gpu

SIZES = [4096, 4097, 8193, 16385, 40001, 65536, 700]


def _edges(kind, n, rng):
    if kind == "random":
        s, d = rng.integers(0, n, 2 * n), rng.integers(0, n, 2 * n)
    elif kind == "sparse":
        s, d = rng.integers(0, n, n // 3), rng.integers(0, n, n // 3)
    else:  # a path through all vertices in random order
        p = rng.permutation(n)
        s, d = p[:-1], p[1:]
    keep = s != d
    return s[keep].astype(np.uint32), d[keep].astype(np.uint32)


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("kind", ["random", "sparse", "path"])
def test_wcc_of_members_split_into_parts(kind, weighted):
    rng = np.random.default_rng(17)
    gs = mk.GraphSet(SIZES, weighted=weighted)
    off = gs.offsets.astype(np.int64)
    mem = [_edges(kind, n, rng) for n in SIZES]
    s = np.concatenate([m[0] + off[i] for i, m in enumerate(mem)])
    d = np.concatenate([m[1] + off[i] for i, m in enumerate(mem)])
    w = to_dev(np.ones(len(s), np.uint32)) if weighted else None
    gs.graph.InsertEdges(to_dev(s), to_dev(d), vals=w)
    assert gs.graph.sync() == 0
    wcc = mk.WCC(gs.graph)
    order = [(int(off[i]), int(off[i + 1])) for i in rng.permutation(len(SIZES))]
    wcc.PrepareRanges(order)
    for _ in range(2):
        wcc.StaticPrepared()
        lab = wcc.Labels().astype(np.int64)
        for i, (ms, md) in enumerate(mem):
            O = OracleGraph(SIZES[i])
            O.insert(ms, md)
            np.testing.assert_array_equal(lab[off[i]:off[i + 1]] - off[i], O.wcc())
    assert gs.graph.sync() == 0


@pytest.mark.parametrize("extra", [[], [70000]])
def test_members_that_outweigh_the_others_are_not_pulled(extra):
    """With a reverse graph and pull levels on, an edge that leaves a heavy
    member is skipped and reported all the same, with and without a member
    too large for shared memory beside it."""
    rng = np.random.default_rng(29)
    sizes = [1500, 60001] + extra + [1100] * 20
    gs = mk.GraphSet(sizes)
    off = gs.offsets.astype(np.int64)
    mem = [_edges("random", n, rng) for n in sizes]
    s = np.concatenate([m[0] + off[i] for i, m in enumerate(mem)])
    d = np.concatenate([m[1] + off[i] for i, m in enumerate(mem)])
    src = [int(m[0][0]) for m in mem]
    want = []
    for i, (ms, md) in enumerate(mem):
        O = OracleGraph(sizes[i])
        O.insert(ms, md)
        want.append(O.bfs(src[i]))
    lost = int(np.flatnonzero(want[0] == want[0].max())[-1])  # a vertex its member does not reach
    assert want[0][lost] > sizes[0]
    reached = want[1] <= sizes[1]
    wide = np.argmax(np.bincount(want[1][reached]))  # the level with the most vertices: a pulled one
    s = np.append(s, off[1] + np.flatnonzero(want[1] == wide)[0])
    d = np.append(d, off[0] + lost)
    rev = mk.DynamicGraph(int(off[-1]), reverse=True)
    gs.graph.InsertEdges(to_dev(s), to_dev(d))
    rev.InsertEdges(to_dev(s), to_dev(d))
    assert gs.graph.sync() == 0 and rev.sync() == 0
    gs.graph.set_tuning(pull_permille=1)
    bfs = mk.BFS(gs.graph, [int(off[i]) + src[i] for i in range(len(sizes))])
    bfs.set_reverse(rev)
    bfs.PrepareMembers([(int(off[i]), int(off[i + 1])) for i in range(len(sizes))])
    bfs.StaticMembers()
    dist = bfs.Distances()
    for i in range(len(sizes)):
        np.testing.assert_array_equal(dist[off[i]:off[i + 1]], want[i])
    with pytest.raises(mk.MeerkatError, match="vertex id out of range"):
        gs.graph.sync()


@pytest.mark.parametrize("weighted", [False, True])
def test_bfs_of_members_that_outweigh_the_others(weighted):
    """One member holds most buckets, so it goes through the device-wide
    kernel beside the others' shared-memory one; levels are each member's
    own, and an edge that leaves the heavy member is skipped and reported."""
    rng = np.random.default_rng(23)
    sizes = [1500, 60001, 1024, 40000] + [1100] * 20
    gs = mk.GraphSet(sizes, weighted=weighted)
    off = gs.offsets.astype(np.int64)
    mem = [_edges("random" if n != 40000 else "sparse", n, rng) for n in sizes]
    s = np.concatenate([m[0] + off[i] for i, m in enumerate(mem)])
    d = np.concatenate([m[1] + off[i] for i, m in enumerate(mem)])
    w = to_dev(np.ones(len(s), np.uint32)) if weighted else None
    gs.graph.InsertEdges(to_dev(s), to_dev(d), vals=w)
    src = [int(m[0][0]) for m in mem]
    bfs = mk.BFS(gs.graph, [int(off[i]) + src[i] for i in range(len(sizes))])
    bfs.PrepareMembers([(int(off[i]), int(off[i + 1])) for i in range(len(sizes))])
    for _ in range(2):
        bfs.StaticMembers()
        dist = bfs.Distances()
        for i, (ms, md) in enumerate(mem):
            O = OracleGraph(sizes[i])
            O.insert(ms, md)
            np.testing.assert_array_equal(dist[off[i]:off[i + 1]], O.bfs(src[i]))
    assert gs.graph.sync() == 0
    out = to_dev(np.array([off[1] + src[1]], np.uint32)), to_dev(np.array([off[0] + 1], np.uint32))
    gs.graph.InsertEdges(*out, vals=to_dev(np.ones(1, np.uint32)) if weighted else None)
    assert gs.graph.sync() == 0
    before = dist[off[0]:off[1]]
    bfs.StaticMembers()
    np.testing.assert_array_equal(bfs.Distances()[off[0]:off[1]], before)
    with pytest.raises(mk.MeerkatError, match="vertex id out of range"):
        gs.graph.sync()


def _layers(depth, n, rng):
    """A source and depth layers of its own, every vertex reached from the layer before."""
    cut = np.concatenate([[0], np.linspace(1, n, depth + 1).astype(int)])
    s = [rng.integers(cut[i], cut[i + 1], cut[i + 2] - cut[i + 1]) for i in range(depth)]
    return np.concatenate(s).astype(np.uint32), np.arange(1, n, dtype=np.uint32)


@pytest.mark.parametrize("weighted", [False, True])
def test_bfs_of_heavy_members_with_many_levels(weighted):
    """Heavy members whose walk ends just before, at and after the level where
    the device-wide kernel gives a member up, one far beyond it, one shallow;
    beside them a member too large for shared memory, as deep, and small ones."""
    rng = np.random.default_rng(31)
    depths = [18, 19, 20, 21, 22, 400]
    mem = [_layers(k, 33000 + 7 * k, rng) for k in depths] + [_edges("random", 50000, rng)]
    mem += [_layers(300, 70000, rng)] + [_edges("random", 700, rng) for _ in range(12)]
    sizes = [33000 + 7 * k for k in depths] + [50000, 70000] + [700] * 12
    gs = mk.GraphSet(sizes, weighted=weighted)
    off = gs.offsets.astype(np.int64)
    s = np.concatenate([m[0] + off[i] for i, m in enumerate(mem)])
    d = np.concatenate([m[1] + off[i] for i, m in enumerate(mem)])
    w = to_dev(np.ones(len(s), np.uint32)) if weighted else None
    gs.graph.InsertEdges(to_dev(s), to_dev(d), vals=w)
    order = rng.permutation(len(sizes))
    src = [int(m[0][0]) for m in mem]
    bfs = mk.BFS(gs.graph, [int(off[i]) + src[i] for i in order])
    bfs.PrepareMembers([(int(off[i]), int(off[i + 1])) for i in order])
    want = []
    for i, (ms, md) in enumerate(mem):
        O = OracleGraph(sizes[i])
        O.insert(ms, md)
        want.append(O.bfs(src[i]))
    for _ in range(2):
        bfs.StaticMembers()
        dist = bfs.Distances()
        for i in range(len(sizes)):
            np.testing.assert_array_equal(dist[off[i]:off[i + 1]], want[i])
    assert gs.graph.sync() == 0
