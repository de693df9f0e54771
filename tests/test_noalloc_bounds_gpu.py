"""The allocation-free entry point where its arrays are just large enough: the support pass's
index headers, one per vertex, share an array sized by pairs of slots, so a graph of as many
vertices as slots is at the edge (with an odd number of slots, past it)."""
import numpy as np
import pytest

from oracle import oracle as O
from sparkx_b200 import gen
import sparkx_b200.pkt as P

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    assert torch.cuda.is_available(), "needs a CUDA device"
    from sparkx_b200 import build
    build.build_engine()
    return torch


def _clique_and_isolated(k, loops, n_extra):
    """K_k (lists of up to k - 1 oriented entries), `loops` self-loops, and isolated vertices until
    there are as many vertices as slots, and `n_extra` more."""
    edges = [(i, j) for i in range(k) for j in range(i + 1, k)] + [(i, i) for i in range(loops)]
    width = k * (k - 1) + loops
    g = gen.from_edges(width + n_extra, edges)
    assert g.width == width and g.n == width + n_extra
    return g


# K_66 has lists of 65 entries (the index starts at 64); 66 * 65 = 4290 = 32 * 134 + 2
@pytest.mark.parametrize("loops,n_extra", [(31, 0), (31, -1), (31, 1), (30, 0), (30, 1), (1, 0), (0, 0), (0, 1)])
def test_as_many_vertices_as_slots(torch_cuda, loops, n_extra):
    torch = torch_cuda
    g = _clique_and_isolated(66, loops, n_extra)
    d_off = torch.from_numpy(np.ascontiguousarray(g.offsets).view(np.int64)).cuda()
    d_nbr = torch.from_numpy(np.ascontiguousarray(g.neighbours, dtype=np.uint32).view(np.int32)).cuda()
    out = torch.full((g.width,), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    P.run_pkt_device_noalloc(d_off.data_ptr(), g.n + 1, d_nbr.data_ptr(), g.width, out.data_ptr())
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy().view(np.uint32), O.pkt(g.offsets, g.neighbours))
