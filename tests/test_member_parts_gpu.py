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
