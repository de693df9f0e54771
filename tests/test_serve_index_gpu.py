"""Served unions keep a rank index of their working rows: built for the first members, for the rows
of every request that joins (behind compacted rows too), and again at each compaction.  Requests of
all row lengths that matter to it (below and at the index's floor, a warp's, one chunk's and
several) join a running union in bursts; results equal the oracle's."""
import os
import time

import numpy as np
import pytest

from conftest import kn, random_graph
from oracle import oracle as O
from sparkx_b200 import gen
import sparkx_b200.pkt as P
from sparkx_b200.serve import PktServer

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def requests():
    import torch
    assert torch.cuda.is_available(), "needs a CUDA device"
    from sparkx_b200 import build
    build.build_engine()
    rng = np.random.default_rng(37)
    gs = [kn(d + 1) for d in (7, 8, 31, 32, 33, 127, 128, 129)]
    gs += [random_graph(rng, n_max=80, self_loop_p=1.0) for _ in range(6)]
    for d in (1023, 1024, 1025, 3000):  # two hubs over a ring: rows of d
        e = [(d, i) for i in range(d)] + [(d + 1, i) for i in range(d)] + [(i, (i + 1) % d) for i in range(d)]
        gs.append(gen.from_edges(d + 2, e))
    gs += [gen.rmat(12, 32, seed=5), gen.rmat(13, 16, seed=6), gen.erdos_renyi(3000, 60_000, 7)]
    return [(g, O.pkt(g.offsets, g.neighbours, threads=4)) for g in gs]


@pytest.fixture(scope="module")
def big():
    g = gen.rmat(19, 16, seed=8)
    return g, O.fast_truss(g.offsets, g.neighbours)[0]


@pytest.mark.parametrize("hash_min,hub_min", [(128, 0), (8, 256), (0, 256), (0, 0)])
def test_joins_behind_a_compacting_union(monkeypatch, requests, big, hash_min, hub_min):
    monkeypatch.setenv("SPARX_SERVE_LANES", "1")
    g, want = big
    P.tuning_clear()
    P.tuning_store(P.tuning_signature(g.offsets), P.PktTuning(hash_min_degree=hash_min, hub_min_degree=hub_min))
    try:
        with PktServer(16 << 30) as srv:
            tb = srv.submit(g.offsets, g.neighbours)
            time.sleep(0.012)
            out = []
            for i in range(0, len(requests), 4):
                out += [(srv.submit(r.offsets, r.neighbours), w) for r, w in requests[i:i + 4]]
                time.sleep(0.004)
            for t, w in out:
                r = srv.wait(t, timeout_ms=120_000)
                assert r.status == P.OK and np.array_equal(r.truss, w)
            r = srv.wait(tb, timeout_ms=120_000)
            assert r.status == P.OK and np.array_equal(r.truss, want)
            # small unions after it, in the same workspace
            out = [(srv.submit(q.offsets, q.neighbours), w) for q, w in requests]
            for t, w in out:
                r = srv.wait(t, timeout_ms=120_000)
                assert r.status == P.OK and np.array_equal(r.truss, w)
            assert srv.info()["joined"] >= 1, srv.info()
    finally:
        P.tuning_clear()


def test_a_request_that_leaves_no_room_for_the_index(monkeypatch, requests):
    """A budget that holds a request's layout and not its index: it is served as before."""
    monkeypatch.setenv("SPARX_SERVE_LANES", "1")
    g, want = requests[-2]

    def serve(budget):
        with PktServer(budget) as srv:
            r = srv.wait(srv.submit(g.offsets, g.neighbours), timeout_ms=60_000)
            return r.status, r.truss

    lo, hi = 1 << 20, 1 << 30
    while hi - lo > 4096:
        mid = (lo + hi) // 2
        lo, hi = (mid, hi) if serve(mid)[0] == P.E_OOM else (lo, mid)
    for budget in (hi, hi + 8192, hi + (1 << 20), hi + (8 << 20)):
        status, truss = serve(budget)
        assert status == P.OK and np.array_equal(truss, want), budget
