"""Static SSSP on a graph large enough for the automatic near-far split.

From 2^20 buckets the threshold doubles when no step is set; hints of 256
edges a vertex put 65,536 vertices above that line."""
import numpy as np
import pytest

import meerkat_b200 as mk
from helpers import to_dev
from meerkat_b200.autotune import SSSP_DELTAS, SSSP_NO_SPLIT
from oracle import OracleGraph

SCALE, V = 16, 1 << 16


def _graph():
    s, d, w = mk.gen_rmat(SCALE, 700000, seed=41, w_lo=1, w_hi=1000)
    G, O = mk.DynamicGraph(V, degree_hints=np.full(V, 256, np.uint32), weighted=True), OracleGraph(V)
    G.InsertEdges(to_dev(s), to_dev(d), vals=to_dev(w))
    O.insert(s, d, w)
    assert G.sync() == 0
    assert G.info()["num_buckets"] > 1 << 20
    return G, O, s, d, int(np.argmax(np.bincount(s, minlength=V)))


@pytest.mark.gpu
def test_automatic_split_matches_oracle_and_can_be_switched_off():
    G, O, s, d, src = _graph()
    sssp = mk.SSSP(G, src, V)
    levels = {}
    for delta in (0, SSSP_NO_SPLIT, 0):
        G.set_tuning(sssp_delta=delta)
        sssp.Static()
        np.testing.assert_array_equal(sssp.Distances(), O.sssp(src))
        assert O.check_parents(src, sssp.packed(), weighted=True) == 0
        levels[delta] = sssp.stats()[0]
    assert levels[0] > levels[SSSP_NO_SPLIT]  # every phase of the split adds levels


@pytest.mark.gpu
def test_automatic_split_in_a_decremental_recompute():
    G, O, s, d, src = _graph()
    G.set_tuning(recompute_permille=1)
    sssp = mk.SSSP(G, src, V)
    sssp.Static()
    es = mk.EdgeSet(V, s, d)
    ds, dd = es.sample_present(len(s) // 5, seed=2)
    tds, tdd = to_dev(ds), to_dev(dd)
    G.DeleteEdges(tds, tdd)
    O.delete(ds, dd)
    sssp.Decremental(tds, tdd)
    assert sssp.decremental_stats()[1]
    np.testing.assert_array_equal(sssp.Distances(), O.sssp(src))
    assert O.check_parents(src, sssp.packed(), weighted=True) == 0


def test_tuner_tries_the_unsplit_form():
    assert SSSP_NO_SPLIT in SSSP_DELTAS and 0 in SSSP_DELTAS
