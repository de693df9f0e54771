"""Waves too small for the whole GPU run in one thread-block cluster, and unions of
up to 32 members are planned by one warp: member counts around that limit,
graphs whose waves stay below, cross and stay above the cluster's bound, with
and without parallel edges, against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O
from sparkx_b200 import gen
from sparkx_b200 import pkt as P

pytestmark = pytest.mark.gpu
O32 = P.PktOptions(out_bits=32)


@pytest.mark.parametrize("count", [1, 2, 31, 32, 33, 70])
def test_member_counts_around_the_warp_planner(count):
    graphs = [gen.rmat(5 + i % 6, 4 + i % 9, seed=100 + i) if i % 3 else gen.erdos_renyi(40 + 7 * i, 300 + 20 * i, i)
              for i in range(count)]
    res = P.run_batch([(g.offsets, g.neighbours) for g in graphs], O32)
    for g, (truss, st, status) in zip(graphs, res):
        want = O.fast_truss(g.offsets, g.neighbours)[0]
        assert status == 0 and np.array_equal(truss, want)
        assert st.k_max == want.max()


@pytest.mark.parametrize("scale,ef", [(6, 8), (9, 16), (11, 16), (13, 16), (15, 12)])
@pytest.mark.parametrize("loop", [P.LOOP_GRAPH, P.LOOP_HOST])
def test_waves_below_and_above_the_bound(scale, ef, loop):
    g = gen.rmat(scale, ef, seed=scale)
    want, st0 = P.run_pkt(g.offsets, g.neighbours, P.PktOptions(out_bits=32, loop=P.LOOP_HOST))
    assert np.array_equal(want, O.fast_truss(g.offsets, g.neighbours)[0])
    got, st = P.run_pkt(g.offsets, g.neighbours, P.PktOptions(out_bits=32, loop=loop))
    assert np.array_equal(got, want)
    assert (st.waves, st.levels, st.peel_edges) == (st0.waves, st0.levels, st0.peel_edges)


def test_parallel_edges_in_small_waves():
    for seed in range(6):
        g = gen.with_parallel_edges(gen.rmat(7 + seed % 3, 8, seed=seed), 0.3, seed=seed)
        got, _ = P.run_pkt(g.offsets, g.neighbours, O32)
        assert np.array_equal(got, O.pkt(g.offsets, g.neighbours))
