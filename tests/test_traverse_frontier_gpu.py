"""GPU: static BFS and SSSP where the frontier queues can go wrong.

A warp queues the vertices that join the next frontier and empties the queue
once it holds enough; what does not fit goes to the frontier directly, and a
vertex with many buckets becomes several work items.  The shapes: one vertex
whose whole neighbourhood is found by few groups (a star), vertices with just
below, at and above one and several work items, and vertex counts around the
32-bit words of the visited bits."""
import numpy as np
import pytest

import meerkat_b200 as mk
from helpers import make_pair

pytestmark = pytest.mark.gpu


def _star(leaves, tail):
    """0 -> every leaf; every 3rd leaf -> the next leaf; a path of `tail`."""
    hub = np.zeros(leaves, np.uint32)
    leaf = np.arange(1, leaves + 1, dtype=np.uint32)
    s = [hub, leaf[:-1:3]]
    d = [leaf, leaf[1::3][: len(leaf[:-1:3])]]
    p = np.arange(leaves, leaves + tail, dtype=np.uint32)
    return leaves + tail + 1, np.concatenate(s + [p]), np.concatenate(d + [p + 1])


def _fans(sizes):
    """0 -> one root per size; root i -> sizes[i] vertices of its own."""
    n = len(sizes)
    s, d, nxt = [np.zeros(n, np.uint32)], [np.arange(1, n + 1, dtype=np.uint32)], n + 1
    for i, k in enumerate(sizes):
        s.append(np.full(k, i + 1, np.uint32))
        d.append(np.arange(nxt, nxt + k, dtype=np.uint32))
        nxt += k
    return nxt, np.concatenate(s), np.concatenate(d)


SHAPES = {"star 31": _star(31, 0), "star 20000": _star(20000, 3), "star 70001": _star(70001, 40),
          "fans": _fans([1, 41, 42, 43, 86, 87, 88, 124, 125, 300, 5000])}


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("shape", list(SHAPES))
def test_static_traversals_on_wide_frontiers(shape, weighted):
    V, s, d = SHAPES[shape]
    w = (np.arange(len(s), dtype=np.uint32) * 7919) % 90 + 1
    G, O = make_pair(V, s, d, w, weighted=weighted)
    bfs = mk.BFS(G, 0, V)
    for _ in range(2):
        bfs.Static()
        np.testing.assert_array_equal(bfs.Distances(), O.bfs(0))
        assert O.check_parents(0, bfs.packed(), weighted=False) == 0
    bfs.set_sources([1, V - 1])
    bfs.Static()
    np.testing.assert_array_equal(bfs.Distances(), np.minimum(O.bfs(1), O.bfs(V - 1)))
    if weighted:
        sssp = mk.SSSP(G, 0, V)
        for _ in range(2):
            sssp.Static()
            np.testing.assert_array_equal(sssp.Distances(), O.sssp(0))
            assert O.check_parents(0, sssp.packed(), weighted=True) == 0
