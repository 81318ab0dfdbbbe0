"""GPU: the range PageRank's two forms against FP64 power iteration.

Runs of at most three iterations push from the slabs, longer ones turn the
edges around and gather in batches of twelve.  The shapes: a hub whose run
fills many whole chunks of 512 pairs, runs that end just below, on and above
a chunk's end, no edge at all, and a skewed graph; the solve ends inside, on
and behind a batch."""
import numpy as np
import pytest

import meerkat_b200 as mk
from helpers import to_dev

pytestmark = pytest.mark.gpu

N = 6000  # vertices of the member; a small one before it moves its first vertex off zero
LEAD = 37


def _into(sizes):
    """sizes[i] in-edges of vertex i, from vertices of its own choice."""
    s = np.concatenate([(np.arange(k) * 7 + i + 1 + np.arange(k) // N) % N for i, k in enumerate(sizes)])
    d = np.repeat(np.arange(len(sizes)), sizes)
    return s, d


def _edges(shape):
    if shape == "none":
        return np.zeros(0, int), np.zeros(0, int)
    if shape == "hub":
        s, d = _into([5999, 2, 1024, 511])
    elif shape == "chunks":  # 511 + 1 + 512 + 513 + 1535 + 31 + 33 ...
        s, d = _into([511, 1, 512, 513, 1535, 31, 33, 32, 64, 480])
    else:
        s, d, _ = mk.gen_rmat(12, 40000, seed=4)
        s, d = s.astype(int), d.astype(int)
    key = np.unique((s.astype(np.int64) * N + d)[s != d])
    return key // N, key % N


def _reference(s, d, iters, damping):
    damping = float(np.float32(damping))  # the entry point takes a 32-bit number
    deg = np.bincount(s, minlength=N)
    pr = np.full(N, 1.0 / N)
    for _ in range(iters):
        nx = np.bincount(d, weights=pr[s] / deg[s], minlength=N)
        pr = (1 - damping) / N + damping * (nx + pr[deg == 0].sum() / N)
    return pr


def _member(s, d, weighted):
    gs = mk.GraphSet([LEAD, N, 5], weighted=weighted)
    if len(s):
        gs.graph.InsertEdges(to_dev(s + LEAD), to_dev(d + LEAD),
                             vals=to_dev(np.ones(len(s))) if weighted else None)
    assert gs.graph.sync() == 0
    return gs


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("shape", ["none", "hub", "chunks", "skewed"])
def test_range_pagerank_forms_match_power_iteration(shape, weighted):
    s, d = _edges(shape)
    gs = _member(s, d, weighted)
    prr = mk.PageRankRange(gs.graph, N)
    for iters in (1, 3, 4, 11, 12, 13, 24, 25):
        prr.Run(LEAD, LEAD + N, 0.85, 1e-30, iters)
        want = _reference(s, d, iters, 0.85)
        # the ranks sum to 1 and are rounded to 24 bits at the end; the rest is FP64
        assert np.abs(prr.Values().astype(np.float64) - want).sum() <= 2.0 ** -24 + 1e-12, iters
    assert gs.graph.sync() == 0


@pytest.mark.parametrize("iters", [2, 30])
@pytest.mark.parametrize("weighted", [False, True])
def test_range_pagerank_reports_an_edge_that_leaves_the_range(weighted, iters):
    """Both forms skip the edge and set the graph's error word."""
    s, d = _edges("skewed")
    gs = _member(s, d, weighted)
    src = LEAD + int(s[0])
    out = to_dev([src, src]), to_dev([3, LEAD + N + 1])  # below and above the range
    gs.graph.InsertEdges(*out, vals=to_dev([1, 1]) if weighted else None)
    prr = mk.PageRankRange(gs.graph, N)
    prr.Run(LEAD, LEAD + N, 0.85, 1e-30, iters)
    assert np.isfinite(prr.Values()).all()
    with pytest.raises(mk.MeerkatError, match="vertex id out of range"):
        gs.graph.sync()


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_range_pagerank_scratch_is_sized_at_creation():
    """No run on a member that has not grown allocates; a fixed scratch stays
    as it is when the member outgrows it, with the same ranks."""
    rng = np.random.default_rng(6)
    key = np.unique(rng.integers(0, N * N, 700000))
    s, d = key // N, key % N
    s, d = s[s != d], d[s != d]
    gs = _member(s, d, False)
    prr = mk.PageRankRange(gs.graph, N)

    def run(reserve=None):
        if reserve is not None:
            prr.reserve(reserve)
        before = _free()
        prr.Run(LEAD, LEAD + N, 0.85, 1e-30, 13)
        assert _free() == before, reserve
        err = np.abs(prr.Values().astype(np.float64) - _reference(s, d, 13, 0.85)).sum()
        assert err <= 2.0 ** -24 + 1e-12, reserve

    run()
    run(len(s))
    run(2000)  # far below the member: pushed from the slabs
    prr.reserve(0)
    free = _free()
    prr.Run(LEAD, LEAD + N, 0.85, 1e-30, 13)
    assert _free() < free  # grown again
    assert gs.graph.sync() == 0
