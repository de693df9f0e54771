"""k-core of graphs full of rows of one entry: a sub-level's elements are dealt out 32 at a time to
the queue entries that own them, and 32 one-entry rows in a row use a whole step up.  Sizes on
both sides of where a warp takes more than one step, in the small waves' cluster (8,192 row
entries) and over the chip (303,104)."""
import numpy as np
import pytest

from oracle import oracle as O
from sparkx_b200 import pkt as P

pytestmark = pytest.mark.gpu


def _csr(n, u, v):
    a, b = np.concatenate([u, v]).astype(np.int64), np.concatenate([v, u]).astype(np.int64)
    key = np.unique(a * n + b)
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    return off, (key % n).astype(np.uint64)


def _star(leaves, hub_last):
    hub = leaves if hub_last else 0
    ids = np.arange(leaves) if hub_last else np.arange(1, leaves + 1)
    return leaves + 1, np.full(leaves, hub), ids


def _clustered(leaves, every, size):
    """Leaves on a clique's members, with a path of `size` after every `every` leaves: runs of one-entry rows
    between longer ones, and both kinds of vertex numbered in turn."""
    u, v, at = [], [], 12
    cu, cv = np.triu_indices(12, 1)
    for i in range(leaves // every):
        ids = np.arange(at, at + every)
        u.append(ids)
        v.append(ids % 12)
        at += every
        p = np.arange(at, at + size - 1)
        u += [p, np.array([at])]
        v += [p + 1, np.array([i % 12])]
        at += size
    return at, np.concatenate([cu] + u), np.concatenate([cv] + v)


def _check(n, u, v):
    off, nbr = _csr(n, u, v)
    want = O.kcore(off, nbr)
    for loop in (P.LOOP_GRAPH, P.LOOP_HOST):
        cores, st = P.run_kcore(off, nbr, P.PktOptions(out_bits=32, loop=loop))
        assert np.array_equal(cores.astype(np.int64), want)
        assert st.levels == np.unique(want[want > 0]).size and st.k_max == want.max()


@pytest.fixture(scope="module", autouse=True)
def _engine():
    from sparkx_b200 import build
    build.build_engine()


@pytest.mark.parametrize("hub_last", [False, True])
@pytest.mark.parametrize("leaves", [31, 33, 8191, 8192, 8193, 8225, 12_000, 16_300, 20_000, 303_104, 303_105, 400_000, 700_001])
def test_stars(leaves, hub_last):
    _check(*_star(leaves, hub_last))


@pytest.mark.parametrize("leaves,every,size", [(9_000, 31, 3), (9_000, 32, 3), (9_000, 33, 2), (9_000, 64, 5), (9_000, 95, 40),
                                               (400_000, 31, 3), (400_000, 32, 2), (400_000, 33, 7), (400_000, 100, 90)])
def test_runs_of_leaves_between_longer_rows(leaves, every, size):
    _check(*_clustered(leaves, every, size))


def test_pairs_and_isolated_vertices():
    n = 900_000
    u = np.arange(0, 600_000, 2)
    _check(n, u, u + 1)
