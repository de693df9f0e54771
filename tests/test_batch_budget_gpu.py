"""A batch holds no more device memory than its budget: a graph that fits it only alone runs
without what is optional (the degree-ordered copy, the rank index), with the same results.

Budgets are found from outside, so no size is repeated here: the least one that runs the graph
at all is its layout, and `support_elements` (the copy's lists are searched from the edge on, so
there are fewer) and `hub_maps` (0 without an index) tell what a run had."""
import numpy as np
import pytest

from oracle import oracle as O
from sparkx_b200 import gen
import sparkx_b200.pkt as P

pytestmark = pytest.mark.gpu
O32 = P.PktOptions(out_bits=32, timeout_ms=120_000)


@pytest.fixture(scope="module")
def member():
    import torch
    assert torch.cuda.is_available(), "needs a CUDA device"
    from sparkx_b200 import build
    build.build_engine()
    g = gen.rmat(13, 16, seed=3)
    P.tuning_clear()
    yield g, O.fast_truss(g.offsets, g.neighbours)[0], P.tuning_signature(g.offsets)
    P.tuning_clear()


def _run(g, budget):
    (truss, st, status), = P.run_batch([(g.offsets, g.neighbours)], O32, hbm_budget_bytes=budget)
    return truss, st, status


def _least(lo, hi, ok):
    """The least budget in (lo, hi] for which ok(budget), to the byte."""
    assert ok(hi)
    while hi - lo > 1:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if ok(mid) else (mid, hi)
    return hi


def _store(key, **knobs):
    P.tuning_store(key, P.PktTuning(hub_min_degree=256, **knobs))


def test_what_is_optional_is_left_out_one_by_one(member):
    g, want, key = member
    big = 8 << 30
    _store(key, relabel=0)
    truss, plain, status = _run(g, big)
    assert status == 0 and np.array_equal(truss, want) and plain.hub_maps > 0
    layout = _least(1 << 20, big, lambda b: _run(g, b)[2] == 0)
    assert _run(g, layout - 1)[2] == P.E_OOM
    truss, st, status = _run(g, layout)
    assert status == 0 and np.array_equal(truss, want) and st.hub_maps == 0
    index = _least(layout, big, lambda b: _run(g, b)[1].hub_maps > 0) - layout

    _store(key, relabel=1)
    truss, copied, status = _run(g, big)
    assert status == 0 and np.array_equal(truss, want) and copied.hub_maps > 0
    assert copied.support_elements < plain.support_elements
    # no room beside the layout: neither
    truss, st, status = _run(g, layout)
    assert status == 0 and np.array_equal(truss, want)
    assert st.hub_maps == 0 and st.support_elements == plain.support_elements
    copy = _least(layout, big, lambda b: _run(g, b)[1].support_elements == copied.support_elements) - layout
    assert index > 0 and copy > 0
    # room for the copy and less than the index more: the copy alone
    for more in (0, index // 2, index - 1):
        truss, st, status = _run(g, layout + copy + more)
        assert status == 0 and np.array_equal(truss, want)
        assert st.hub_maps == 0 and st.support_elements == copied.support_elements, more
    # room for both
    truss, st, status = _run(g, layout + copy + index)
    assert status == 0 and np.array_equal(truss, want)
    assert st.hub_maps > 0 and st.support_elements == copied.support_elements


def test_several_members_in_a_tight_budget(member):
    """Members packed one to a union: each runs without the copy where the budget is its layout."""
    g, want, key = member
    _store(key, relabel=1)
    layout = _least(1 << 20, 8 << 30, lambda b: _run(g, b)[2] == 0)
    for budget in (layout, layout + 4096):
        for truss, st, status in P.run_batch([(g.offsets, g.neighbours)] * 3, O32, hbm_budget_bytes=budget):
            assert status == 0 and np.array_equal(truss, want)
            assert st.hub_maps == 0
