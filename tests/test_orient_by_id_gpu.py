"""Degree-ordered copies are oriented by id and their support pass searches only
the entries after an edge's own: list tails around the runs of 24 and the groups
of 32, empty tails, self-loops (in the middle of a row, first and last), unions,
and each way a list is searched, against the decomposition on the caller's ids."""
import numpy as np
import pytest

from conftest import kn
from sparkx_b200 import gen
from sparkx_b200 import pkt as P

pytestmark = pytest.mark.gpu
O32 = P.PktOptions(out_bits=32)
SEARCHES = [dict(), dict(sample_min=8), dict(sample_min=4096), dict(sup_hash_min=4), dict(support_kernel=2)]


def _run(g, **tuning):
    key = P.tuning_signature(g.offsets)
    try:
        P.tuning_store(key, P.PktTuning(**tuning))
        out, st = P.run_pkt(g.offsets, g.neighbours, O32)
        assert P.tuning_last() == (P.PktTuning(**tuning), key)
        return out, st
    finally:
        P.tuning_clear()


@pytest.mark.parametrize("k", [2, 3, 24, 25, 26, 32, 33, 34, 57, 66, 130, 300])
def test_cliques(k):
    g = kn(k)  # every tail length from 0 to k - 1, all ids in one degree bucket
    for s in SEARCHES:
        got, st = _run(g, relabel=1, **s)
        assert np.all(got == k) and st.triangles == k * (k - 1) * (k - 2) // 6


@pytest.mark.parametrize("scale,ef", [(6, 2), (9, 20), (12, 16), (14, 8)])
@pytest.mark.parametrize("loops", [False, True])
def test_skewed_graphs(scale, ef, loops):
    g = gen.rmat(scale, ef, seed=scale + ef)
    if loops:
        n = len(g.offsets) - 1
        src = np.repeat(np.arange(n), np.diff(np.asarray(g.offsets).astype(np.int64)))
        edges = list(zip(src.tolist(), np.asarray(g.neighbours).tolist()))
        g = gen.from_edges(n, edges + [(u, u) for u in range(0, n, 3)])
    want, st0 = _run(g, relabel=0)
    for s in SEARCHES:
        got, st = _run(g, relabel=1, **s)
        assert np.array_equal(got, want), s
        assert (st.triangles, st.max_support) == (st0.triangles, st0.max_support), s


def test_union():
    members = [gen.rmat(11, 16, seed=1), kn(40), gen.erdos_renyi(3000, 40000, 2), gen.from_edges(3, [(0, 1)]),
               gen.rmat(12, 8, seed=4)]
    pairs = [(m.offsets, m.neighbours) for m in members]
    want = [P.run_pkt(o, x, O32)[0] for o, x in pairs]
    P.run_batch(pairs, O32)
    key = P.tuning_last()[1]
    for s in SEARCHES:
        P.tuning_store(key, P.PktTuning(relabel=1, **s))
        try:
            res = P.run_batch(pairs, O32)
        finally:
            P.tuning_clear()
        for w, (got, _, status) in zip(want, res):
            assert status == 0 and np.array_equal(got, w), s


@pytest.mark.parametrize("d", [31, 32, 33, 127, 128, 129, 257, 2047, 2048, 2049, 3073, 20_000])
def test_row_lengths_of_the_copy(d):
    """Two hubs with rows of d (a warp's, a block's, parts of both) over a ring of mixed degrees."""
    ring = np.arange(d)
    edges = [(d, i) for i in range(d)] + [(d + 1, i) for i in range(0, d, 2)] + [(int(i), int((i + 1) % d)) for i in ring]
    edges += [(int(i), int((i + k) % d)) for i in ring[::7] for k in range(2, 9)]
    edges += [(u, v) for u in range(d + 2, d + 14) for v in range(d + 2, u)] + [(d, d + 1)]
    g = gen.from_edges(d + 14, [(u, v) for u, v in edges if u != v])
    want, st0 = _run(g, relabel=0)
    got, st = _run(g, relabel=1)
    assert np.array_equal(got, want) and st.triangles == st0.triangles


@pytest.mark.parametrize("scale,ef,relabels", [(17, 16, 0), (19, 6, 0), (19, 18, 1)])
def test_rule_for_keys_without_an_entry(scale, ef, relabels):
    g = gen.rmat(scale, ef, seed=11)
    P.tuning_clear()
    got, st = P.run_pkt(g.offsets, g.neighbours, O32)
    used, key = P.tuning_last()
    assert used.relabel == relabels == int(key[0] >= 23 and key[2] >= 4)
    want, st0 = _run(g, relabel=1 - relabels)
    assert np.array_equal(got, want) and st.triangles == st0.triangles
