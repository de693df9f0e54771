"""Clustering coefficients of vertices whose rows lie at the edges of the lane, warp and
block forms (32, 2048 entries, and the four slots read at a time), with simple and with
parallel edges, against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O
from sparkx_b200 import pkt as P

pytestmark = pytest.mark.gpu
RTOL = 1e-12  # the averages are sums of doubles in another order


def _wheel(d, parallel):
    """A hub with a ring of d vertices, and a second hub on every third of them."""
    ring = np.arange(d, dtype=np.int64)
    a = np.concatenate([np.full(d, d), ring, np.full((d + 2) // 3, d + 1)])
    b = np.concatenate([ring, (ring + 1) % d, ring[::3]])
    if parallel:
        a, b = np.concatenate([a, a[::5]]), np.concatenate([b, b[::5]])
    src, dst = np.concatenate([a, b]), np.concatenate([b, a])
    order = np.lexsort((dst, src))
    off = np.zeros(d + 3, dtype=np.uint64)
    np.cumsum(np.bincount(src, minlength=d + 2), out=off[1:])
    return off, dst[order].astype(np.uint64)


@pytest.mark.parametrize("d", [4, 31, 32, 33, 127, 128, 129, 2047, 2048, 2049, 3073, 20_000])
@pytest.mark.parametrize("parallel", [False, True])
def test_row_lengths(d, parallel):
    off, nbr = _wheel(d, parallel)
    local, trans, avg, _ = P.run_clustering(off, nbr)
    want_local, want_trans, want_avg = O.clustering(off, nbr)
    assert np.array_equal(local, want_local)
    assert trans == pytest.approx(want_trans, rel=RTOL, abs=0)
    assert avg == pytest.approx(want_avg, rel=RTOL, abs=0)
