"""Device inputs are checked in one pass: neighbour arrays at every 4-byte
alignment, widths around the four-at-a-time loads, and a defect in the first,
last and odd places, each refused as before and without harm to the next call."""
import numpy as np
import pytest

from oracle import oracle as O
from sparkx_b200 import gen
from sparkx_b200 import pkt as P

pytestmark = pytest.mark.gpu


def _run(off, nbr, shift=0):
    import torch
    d_off = torch.from_numpy(off.astype(np.int64)).cuda()
    buf = torch.zeros(nbr.shape[0] + 8, dtype=torch.int32, device="cuda")
    d_nbr = buf[shift:shift + nbr.shape[0]]
    d_nbr.copy_(torch.from_numpy(nbr.astype(np.int64).astype(np.int32)))
    out = torch.empty(nbr.shape[0] + 1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    P.run_pkt_device(d_off.data_ptr(), off.shape[0], d_nbr.data_ptr(), nbr.shape[0], out.data_ptr(),
                     P.PktOptions(out_bits=32))
    return out[:nbr.shape[0]].cpu().numpy().astype(np.uint32)


@pytest.mark.parametrize("shift", [0, 1, 2, 3])
@pytest.mark.parametrize("edges", [1, 2, 3, 4, 5, 300])
def test_alignments_and_widths(shift, edges):
    g = gen.erdos_renyi(60, edges, edges)
    assert np.array_equal(_run(g.offsets, g.neighbours, shift), O.pkt(g.offsets, g.neighbours))


@pytest.mark.parametrize("shift", [0, 1])
def test_defects_are_refused(shift):
    g = gen.rmat(9, 8, seed=3)
    w = g.width
    want = O.pkt(g.offsets, g.neighbours)
    for at in (0, 1, 5, w // 2, w - 2, w - 1):
        bad = g.neighbours.copy()
        bad[at] = g.n
        with pytest.raises(P.PktError) as e:
            _run(g.offsets, bad, shift)
        assert e.value.status == P.E_INVALID_CSR
    for at, value in ((0, 1), (1, w + 1), (g.n // 2, w), (g.n, w - 1), (g.n, w + 1)):
        off = g.offsets.copy()
        off[at] = value
        with pytest.raises(P.PktError) as e:
            _run(off, g.neighbours, shift)
        assert e.value.status == P.E_INVALID_CSR
    assert np.array_equal(_run(g.offsets, g.neighbours, shift), want)
