"""GPU: static triangle counts where the staged lists change form.

In a complete graph on n vertices the oriented lists have every length from 0
to n - 1, so the sizes below cross the buckets of a staged set (16, 32, ...,
512 of four slots), its last half-empty and over-full sizes, and the limit of
1,024 entries from which a block takes the vertex; with a fringe of pendant
vertices and of triangles hung on single vertices."""
import numpy as np
import pytest

import meerkat_b200 as mk
from helpers import degree_hints, symmetrise, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("n", [2, 3, 9, 17, 33, 130, 257, 513, 1025, 1090])
def test_triangles_of_a_clique_with_a_fringe(n, weighted):
    a, b = np.triu_indices(n, 1)
    base, tri = n, n + n  # pendant i - (n + i); a triangle on every 5th vertex
    i = np.arange(n)
    hung = i[::5]
    t0 = tri + 2 * np.arange(len(hung))
    s = np.concatenate([a, i, hung, hung, t0])
    d = np.concatenate([b, base + i, t0, t0 + 1, t0 + 1])
    V = tri + 2 * len(hung)
    ss, sd = symmetrise(s.astype(np.uint32), d.astype(np.uint32))
    G = mk.DynamicGraph(V, degree_hints=degree_hints(ss, V), weighted=weighted)
    G.InsertEdges(to_dev(ss), to_dev(sd), vals=to_dev(np.ones(len(ss), np.uint32)) if weighted else None)
    tc = mk.TC(G, V)
    for _ in range(2):
        tc.Static()
        assert tc.GetCount() == n * (n - 1) * (n - 2) // 6 + len(hung)
