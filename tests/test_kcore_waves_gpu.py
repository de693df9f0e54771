"""Sub-levels of the k-core peel spread over their row entries: hub rows around a
warp's 32 entries and around the bound of the small waves' cluster (16,384),
frontiers of many short rows, and hubs that hang on one another."""
import numpy as np
import pytest

from oracle import oracle as O
from sparkx_b200 import pkt as P

pytestmark = pytest.mark.gpu


def _csr(n, a, b):
    src, dst = np.concatenate([a, b]), np.concatenate([b, a])
    order = np.lexsort((dst, src))
    off = np.zeros(n + 1, dtype=np.uint64)
    np.cumsum(np.bincount(src, minlength=n), out=off[1:])
    return off, dst[order].astype(np.uint64)


def _check(off, nbr):
    for mode, oracle_mode in ((P.SUPPORT_WIDE, O.MODE_WIDE), (P.SUPPORT_U8, O.MODE_U8)):
        want = O.kcore(off, nbr, mode=oracle_mode)
        for loop in (P.LOOP_GRAPH, P.LOOP_HOST):
            got, _ = P.run_kcore(off, nbr, P.PktOptions(out_bits=32, support_mode=mode, loop=loop))
            assert np.array_equal(got, want), (mode, loop)


@pytest.mark.parametrize("leaves", [1, 31, 32, 33, 255, 256, 16383, 16384, 16385, 60000])
def test_stars(leaves):
    # a star, and two hubs that share every leaf and an edge (core 2)
    a = np.concatenate([np.zeros(leaves, np.int64), np.full(leaves, leaves + 1), np.full(leaves, leaves + 2),
                        [leaves + 1]])
    two = leaves + 3 + np.arange(leaves)
    b = np.concatenate([1 + np.arange(leaves), two, two, [leaves + 2]])
    _check(*_csr(2 * leaves + 3, a, b))


@pytest.mark.parametrize("n", [4000, 20000, 40000])
def test_many_short_rows_at_once(n):
    # a cycle with chords to a clique of 40: whole levels fall in one wave
    v = np.arange(n)
    a = np.concatenate([v, v, np.repeat(n + np.arange(40), 40)])
    b = np.concatenate([(v + 1) % n, n + v % 40, np.tile(n + np.arange(40), 40)])
    keep = a != b
    lo, hi = np.minimum(a, b)[keep], np.maximum(a, b)[keep]
    pairs = np.unique(lo * (n + 40) + hi)
    _check(*_csr(n + 40, pairs // (n + 40), pairs % (n + 40)))
