"""A served request that is run again by itself (another one in its union had a defect) stays
within its lane's budget: the degree-ordered copy and the rank index, each of which fits beside the
layout, are not both taken where they do not fit together."""
import numpy as np
import pytest

from test_batch_budget_gpu import O32, _least, _run, _store, member  # noqa: F401 (a fixture)
import sparkx_b200.pkt as P
from sparkx_b200.serve import PktServer

pytestmark = pytest.mark.gpu
BAD = (np.array([0, 1, 3, 4, 4], np.uint64), np.array([1, 0, 2, 3], np.uint32))


def test_rerun_requests_stay_within_the_lane(monkeypatch, member):  # noqa: F811
    monkeypatch.setenv("SPARX_SERVE_LANES", "1")
    g, want, key = member
    big = 8 << 30
    _store(key, relabel=0)
    layout = _least(1 << 20, big, lambda b: _run(g, b)[2] == 0)
    index = _least(layout, big, lambda b: _run(g, b)[1].hub_maps > 0) - layout
    _store(key, relabel=1)
    copied = _run(g, big)[1].support_elements
    copy = _least(layout, big, lambda b: _run(g, b)[1].support_elements == copied) - layout
    main = layout + index + (1 << 20)  # a served union's layout (room for 4,096 members) and the index
    assert layout + copy < main < layout + copy + index
    # a lane keeps a fifth of its budget for preparing joins
    with PktServer(main * 5 // 4 + 4, P.PktOptions(out_bits=32)) as srv:
        for _ in range(200):
            tb, tg = srv.submit(*BAD), srv.submit(g.offsets, g.neighbours)
            rb, rg = srv.wait(tb, timeout_ms=60_000), srv.wait(tg, timeout_ms=60_000)
            assert rb.status == P.E_INVALID_CSR
            assert rg.status == P.OK and np.array_equal(rg.truss, want)
            if rg.stats.support_elements:  # run again by itself: a served result carries no such count
                break
        else:
            pytest.skip("the two requests never shared a union")
    assert rg.stats.support_elements == copied
    assert rg.stats.hub_maps == 0
