"""The peel's row compaction at the edges of its tiles (8,192 slots) and of its
32-slot words: a graph large enough to compact (2^20 slots) with its slot count
moved by single pendant edges, isolated vertices at the end (rows that start at
the array's end), and tuned fills that compact often and rarely."""
import numpy as np
import pytest

from oracle import oracle as O
from sparkx_b200 import gen
from sparkx_b200 import pkt as P

pytestmark = pytest.mark.gpu
O32 = P.PktOptions(out_bits=32)


@pytest.fixture(scope="module")
def base():
    g = gen.rmat(16, 12, seed=31)
    return g, O.fast_truss(g.offsets, g.neighbours)[0]


def _with_leaves(g, truss, leaves, isolated):
    """`leaves` new vertices hanging off vertices 0, 1, ..., and `isolated` ones behind them."""
    n = g.n
    src = np.repeat(np.arange(n, dtype=np.int64), np.diff(g.offsets.astype(np.int64)))
    at, new = np.arange(leaves) % n, n + np.arange(leaves)
    a = np.concatenate([src, at, new])
    b = np.concatenate([g.neighbours.astype(np.int64), new, at])
    t = np.concatenate([truss, np.full(2 * leaves, 2, dtype=truss.dtype)])
    order = np.lexsort((b, a))
    off = np.zeros(n + leaves + isolated + 1, dtype=np.uint64)
    np.cumsum(np.bincount(a, minlength=n + leaves + isolated), out=off[1:])
    return off, b[order].astype(np.uint64), t[order]


@pytest.mark.parametrize("past", [0, 2, 30, 32, 34, 8190])
@pytest.mark.parametrize("isolated", [0, 5])
def test_slot_counts_around_words_and_tiles(base, past, isolated):
    g, truss = base
    leaves = (-g.width % 8192 + past) // 2
    off, nbr, want = _with_leaves(g, truss, leaves, isolated)
    assert nbr.shape[0] % 8192 == past and nbr.shape[0] >= 1 << 20
    got, st = P.run_pkt(off, nbr, O32)
    assert st.compactions >= 1 and np.array_equal(got, want)


@pytest.mark.parametrize("pct", [10, 50, 99, 100])
def test_fills(base, pct):
    g, truss = base
    key = P.tuning_signature(g.offsets)
    try:
        P.tuning_store(key, P.PktTuning(compact_pct=pct))
        got, _ = P.run_pkt(g.offsets, g.neighbours, O32)
    finally:
        P.tuning_clear()
    assert np.array_equal(got, truss)
