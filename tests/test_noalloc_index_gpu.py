"""The allocation-free entry point's rank index: rows of every length that matters to it, calls one
after another over the same scratch, and graphs on both sides of what the scratch holds with the
index (60 bytes a slot, 20 a vertex) and at all (44 and 12)."""
import numpy as np
import pytest

from conftest import kn, random_graph
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


def _run(torch, g):
    d_off = torch.from_numpy(np.ascontiguousarray(g.offsets).view(np.int64)).cuda()
    d_nbr = torch.from_numpy(np.ascontiguousarray(g.neighbours, dtype=np.uint32).view(np.int32)).cuda()
    out = torch.full((max(1, g.width),), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    P.run_pkt_device_noalloc(d_off.data_ptr(), g.n + 1, d_nbr.data_ptr(), g.width, out.data_ptr())
    torch.cuda.synchronize()
    return out.cpu().numpy().view(np.uint32)[: g.width]


def _hubs(d, loops=0):
    """Two hubs joined to a ring of d vertices, `loops` of which carry a self-loop."""
    e = [(d, i) for i in range(d)] + [(d + 1, i) for i in range(d)] + [(i, (i + 1) % d) for i in range(d)]
    return gen.from_edges(d + 2, e + [(i, i) for i in range(loops)])


def test_row_lengths(torch_cuda):
    rng = np.random.default_rng(47)
    graphs = [kn(d + 1) for d in (30, 31, 32, 33, 63, 64, 127, 128, 129, 257)]
    graphs += [_hubs(d, loops) for d, loops in ((127, 5), (128, 0), (1023, 9), (1024, 0), (1025, 0), (3000, 100))]
    graphs += [random_graph(rng, n_max=90, self_loop_p=1.0) for _ in range(10)]
    graphs += [gen.rmat(14, 16, seed=3), gen.from_edges(5, []), gen.rmat(13, 40, seed=4), gen.from_edges(3, [(0, 1)])]
    for g in graphs + graphs[::3]:
        assert np.array_equal(_run(torch_cuda, g), O.pkt(g.offsets, g.neighbours, threads=4)), (g.n, g.width)


@pytest.mark.parametrize("m", [540_000, 552_000, 560_000, 620_000, 750_000])
def test_around_what_the_scratch_holds(torch_cuda, m):
    g = gen.erdos_renyi(6000, m, 9)
    assert np.array_equal(_run(torch_cuda, g), O.pkt(g.offsets, g.neighbours, threads=8))


def test_skewed_graph_without_the_index(torch_cuda):
    g = gen.rmat(16, 12, seed=5)
    assert 60 * g.width + 20 * g.n > 64 << 20 > 44 * g.width + 12 * g.n + (1 << 18)
    assert np.array_equal(_run(torch_cuda, g), O.fast_truss(g.offsets, g.neighbours)[0])
