"""The support pass's pair form (a thread per edge, every oriented list of at most 64
entries) around its bounds: list lengths up to, at and past 64, equal and empty
lists, parallel edges; supports and truss numbers against the explicit balanced
and vertex forms, cliques against their known answers."""
import numpy as np
import pytest

from conftest import kn
from sparkx_b200 import gen
from sparkx_b200 import pkt as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [2, 3, 4, 33, 64, 65, 66, 67])
def test_cliques_around_the_list_bound(k):
    g = kn(k)  # oriented lists of 0 to k - 1 entries
    sup, st = P.run_triangles(g.offsets, g.neighbours)
    assert np.all(sup == k - 2) and st.triangles == k * (k - 1) * (k - 2) // 6


@pytest.mark.parametrize("n,m", [(50, 40), (1000, 3000), (3000, 60000), (4000, 200000), (2000, 120000)])
def test_forms_agree(n, m):
    for g in (gen.erdos_renyi(n, m, n + m), gen.rmat(max(6, n.bit_length() - 1), max(2, m // n), seed=m)):
        got, st = P.run_triangles(g.offsets, g.neighbours)
        for form in (1, 2):
            want, st1 = P.run_triangles(g.offsets, g.neighbours, P.PktOptions(support_kernel=form))
            assert np.array_equal(got, want) and st.triangles == st1.triangles


def test_parallel_edges():
    for seed in range(5):
        g = gen.with_parallel_edges(gen.erdos_renyi(400, 2500, seed), 0.3, seed=seed)
        got, _ = P.run_triangles(g.offsets, g.neighbours)
        want, _ = P.run_triangles(g.offsets, g.neighbours, P.PktOptions(support_kernel=1))
        assert np.array_equal(got, want)
