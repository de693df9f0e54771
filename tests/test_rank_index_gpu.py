"""The rank index of sorted lists (the search of the support pass) at the sizes
where it can go wrong: list lengths around every power of two, lists longer
than a warp's row (2048), ids clustered so that many entries share a bucket,
and lists below and above the index's floor.  Cliques give the answers:
every edge of K_k lies in k - 2 triangles and has truss number k."""
import numpy as np
import pytest

from sparkx_b200 import gen
from sparkx_b200 import pkt as P

pytestmark = pytest.mark.gpu
O32 = P.PktOptions(out_bits=32)


def _clique(ids, n, leaves=0):
    """CSR over n vertices: K_k on `ids`, and `leaves` vertices hanging off ids[0] (the remaining
    vertices, in order, so that its row spans the whole id range)."""
    ids = np.sort(np.asarray(ids, dtype=np.int64))
    k = ids.shape[0]
    a, b = np.repeat(ids, k), np.tile(ids, k)
    keep = a != b
    rest = np.setdiff1d(np.arange(n), ids)[:leaves]
    src = np.concatenate([a[keep], np.full(rest.shape, ids[0]), rest])
    dst = np.concatenate([b[keep], rest, np.full(rest.shape, ids[0])])
    order = np.lexsort((dst, src))
    src, dst = src[order], dst[order]
    off = np.zeros(n + 1, dtype=np.uint64)
    np.cumsum(np.bincount(src, minlength=n), out=off[1:])
    inside = np.isin(src, ids) & np.isin(dst, ids)
    return off, dst.astype(np.uint64), np.where(inside, k, 2)


def _check(off, nbr, truss, tuning=None):
    key = P.tuning_signature(off)
    try:
        if tuning is not None:
            P.tuning_store(key, tuning)
        got, st = P.run_pkt(off, nbr, O32)
        sup, _ = P.run_triangles(off, nbr)
    finally:
        P.tuning_clear()
    assert np.array_equal(sup, truss - 2)
    assert np.array_equal(got, truss)


@pytest.mark.parametrize("k", [7, 8, 9, 10, 16, 17, 18, 33, 64, 65, 66, 129, 130, 513, 2049, 2050, 2200])
def test_list_lengths(k):
    # the oriented lists of K_k have every length from 0 to k - 1
    _check(*_clique(np.arange(k), k), P.PktTuning(sample_min=8, hash_min_degree=8, hub_min_degree=0))


@pytest.mark.parametrize("k", [40, 300])
@pytest.mark.parametrize("spread", ["two_clusters", "tail", "even", "head_and_leaves"])
def test_clustered_ids(k, spread):
    n = 200_000
    ids = {"two_clusters": np.concatenate([np.arange(k // 2), n - 1 - np.arange(k - k // 2)]),
           "tail": n - 1 - np.arange(k), "even": np.arange(k) * (n // k),
           "head_and_leaves": np.arange(k)}[spread]
    leaves = n - k if spread == "head_and_leaves" else 3000
    off, nbr, truss = _clique(ids, n, leaves)
    _check(off, nbr, truss, P.PktTuning(sample_min=8, hash_min_degree=8))
    _check(off, nbr, truss)


def test_floor_below_and_above_every_list():
    g = gen.rmat(13, 16, seed=21)
    want, _ = P.run_triangles(g.offsets, g.neighbours)
    for floor in (2, 8, 9, 31, 64, 65, 1 << 20):
        key = P.tuning_signature(g.offsets)
        try:
            P.tuning_store(key, P.PktTuning(sample_min=floor))
            got, _ = P.run_triangles(g.offsets, g.neighbours)
        finally:
            P.tuning_clear()
        assert np.array_equal(got, want), floor
