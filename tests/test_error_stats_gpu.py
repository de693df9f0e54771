"""What a call's stats say when its input is refused before any row is read (an id out of range,
offsets that decrease): nothing was counted, whatever an earlier call left in the workspace."""
import ctypes

import numpy as np
import pytest

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


def _bad_id(g):
    nbr = np.ascontiguousarray(g.neighbours).copy()
    nbr[g.width // 2] = g.n + 5
    return np.ascontiguousarray(g.offsets), nbr


def _decreasing(g):
    off = np.ascontiguousarray(g.offsets).copy()
    off[g.n // 2] = off[g.n // 2 + 1] + np.uint64(1)
    return off, np.ascontiguousarray(g.neighbours)


@pytest.mark.parametrize("spoil", [_bad_id, _decreasing])
@pytest.mark.parametrize("entry", ["run", "run_u32", "triangles", "clustering", "device"])
def test_nothing_is_counted(torch_cuda, entry, spoil):
    torch, L = torch_cuda, P.lib()
    g = gen.rmat(10, 16, seed=3)
    P.run_pkt(g.offsets, g.neighbours, P.PktOptions(out_bits=32))  # leaves its counts in the workspace
    off, nbr = spoil(g)
    o, st = P.PktOptions(out_bits=32).c(), P._Stats()
    refs = ctypes.byref(o), ctypes.byref(st)
    out = np.zeros(g.width, np.uint32)
    if entry == "device":
        d_off, d_nbr = torch.from_numpy(off.view(np.int64)).cuda(), torch.from_numpy(nbr.astype(np.uint32).view(np.int32)).cuda()
        d_out = torch.zeros(g.width, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        rc = L.sparx_pkt_run_device(d_off.data_ptr(), g.n + 1, d_nbr.data_ptr(), g.width, d_out.data_ptr(), *refs, None)
    elif entry == "run_u32":
        nbr = nbr.astype(np.uint32)
        rc = L.sparx_pkt_run_u32(off.ctypes.data, g.n + 1, nbr.ctypes.data, g.width, out.ctypes.data, *refs)
    else:
        nbr = nbr.astype(np.uint64)
        a = off.ctypes.data, g.n + 1, nbr.ctypes.data, g.width
        if entry == "run":
            rc = L.sparx_pkt_run(*a, out.ctypes.data, *refs)
        elif entry == "triangles":
            rc = L.sparx_triangles_run(*a, out.ctypes.data, *refs)
        else:
            local, t, m = np.zeros(g.n), ctypes.c_double(), ctypes.c_double()
            rc = L.sparx_clustering_run(*a, local.ctypes.data, ctypes.byref(t), ctypes.byref(m), *refs)
    assert rc == P.E_INVALID_CSR
    assert (st.n, st.width) == (g.n, g.width)
    assert (st.m, st.self_loops, st.triangles, st.waves, st.k_max) == (0, g.width, 0, 0, 0)
