"""Timed cases of the framework's public entry points, from the smallest calls to the largest.

Graphs are those of the configurations the framework is built for: Erdos-Renyi, R-MAT
(a, b, c = 0.57, 0.19, 0.19, edge factor 16), a 21-mer de Bruijn graph and the batched mix
(n log-uniform in 10^3..10^6, average degree log-uniform in 4..64, half ER, half R-MAT).
They are generated on the GPU from the seed alone; entry points that take host arrays get
host arrays, in the reference's u64 layout unless said otherwise.
"""
import math

import numpy as np
import torch

from sparkx_b200 import pkt

DEV = "cuda"
_RMAT_ABC = (0.57, 0.19, 0.19)


def listed():
    return [
        # the smallest call: a graph of a thousand vertices, device arrays in and out
        {"name": "pkt_er_1k", "op": "pkt", "graph": "er", "n": 1000, "m": 4000},
        # a small social-style graph: hundreds of short peel waves, latency only
        {"name": "pkt_rmat_12", "op": "pkt", "graph": "rmat", "n": 1 << 12, "m": 48_000},
        # sparse random graph of 10^5 vertices, 10^6 edges: few triangles, a handful of waves
        {"name": "pkt_er_100k", "op": "pkt", "graph": "er", "n": 100_000, "m": 1_000_000},
        # a mid-size skewed graph (15 M slots): every phase counts
        {"name": "pkt_rmat_19", "op": "pkt", "graph": "rmat", "n": 1 << 19, "m": 7_700_000},
        # the headline workload: 128 M slots, 2.1 G triangles
        {"name": "pkt_rmat_22", "op": "pkt", "graph": "rmat", "n": 1 << 22, "m": 64_000_000},
        # 21-mer de Bruijn graph of a 20 Mbase sequence: 49 M slots of degree about 2, a few dozen triangles
        {"name": "pkt_debruijn", "op": "pkt", "graph": "dbg", "n": 26_000_000, "m": 24_700_000},
        # the drop-in call: host u64 arrays in, one byte per slot out
        {"name": "pkt_host_rmat_16", "op": "pkt_host", "graph": "rmat", "n": 1 << 16, "m": 900_000, "bits": 8},
        # triangle support per slot (host arrays)
        {"name": "triangles_rmat_20", "op": "triangles", "graph": "rmat", "n": 1 << 20, "m": 15_600_000},
        # clustering coefficients (host arrays, f64 out)
        {"name": "clustering_rmat_17", "op": "clustering", "graph": "rmat", "n": 1 << 17, "m": 1_850_000},
        # core numbers (host arrays)
        {"name": "kcore_rmat_20", "op": "kcore", "graph": "rmat", "n": 1 << 20, "m": 15_600_000},
        # a batch of independent graphs in one call (host u32 ids)
        {"name": "batch_mix_24", "op": "batch", "graph": "mix", "count": 24, "n_lo": 1000, "n_hi": 1_000_000},
        # MatrixMarket text to CSR
        {"name": "mtx_rmat_17", "op": "mtx", "graph": "rmat", "n": 1 << 17, "m": 1_850_000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["pkt", "pkt", "pkt", "pkt_host", "triangles", "clustering", "kcore", "batch", "mtx"])
    if op == "batch":
        return {"op": op, "graph": "mix", "count": rng.randint(2, 24), "n_lo": rng.randint(500, 2000),
                "n_hi": _log_int(rng, 3000, 1_000_000)}
    kind = rng.choice(["er", "rmat", "rmat", "dbg"]) if op == "pkt" else rng.choice(["er", "rmat", "rmat"])
    if kind == "dbg":
        n = _log_int(rng, 200_000, 26_000_000)
        return {"op": op, "graph": "dbg", "n": n, "m": int(n * 0.95)}
    if kind == "er":
        n = _log_int(rng, 1000, 1_000_000 if op == "pkt" else 300_000)
        m = int(n * rng.uniform(2.0, 24.0))
    else:
        top = {"pkt": 21, "pkt_host": 16, "triangles": 20, "clustering": 19, "kcore": 20, "mtx": 17}[op]
        n = 1 << rng.randint(10, top)
        m = int(n * rng.uniform(4.0, 13.0))
    case = {"op": op, "graph": kind, "n": n, "m": m}
    if op == "pkt_host":
        case["bits"] = rng.choice([8, 32])
    return case


# ---- inputs ------------------------------------------------------------------------------


def _csr(n, pairs):
    """Symmetric CSR (i64 offsets, i64 neighbours, sorted rows) of the distinct pairs lo * n + hi."""
    lo, hi = pairs // n, pairs % n
    slots = torch.cat([pairs, hi * n + lo]).sort().values
    off = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(torch.bincount(slots // n, minlength=n), 0, out=off[1:])
    return off, slots % n


def _pairs(n, a, b):
    """Distinct pairs {a, b}, a != b, as min * n + max."""
    keep = a != b
    a, b = a[keep], b[keep]
    return torch.unique(torch.minimum(a, b) * n + torch.maximum(a, b))


def _exactly(pairs, m, g):
    """m of the pairs, drawn evenly: a graph's size depends on its parameters, not on its seed."""
    if pairs.numel() < m:
        raise ValueError(f"{pairs.numel()} distinct pairs, {m} are wanted")
    return pairs[torch.randperm(pairs.numel(), device=DEV, generator=g)[:m]]


def _distinct(n, m, g, draw_pairs):
    pairs, more = torch.empty(0, dtype=torch.int64, device=DEV), m + m // 16 + 16
    while pairs.numel() < m:
        u, v = draw_pairs(more)
        pairs = torch.unique(torch.cat([pairs, _pairs(n, u, v)]))
        more = max(2 * (m - pairs.numel()), m // 16 + 16)
    return _csr(n, _exactly(pairs, m, g))


def _er(n, m, g):
    return _distinct(n, m, g, lambda k: torch.randint(n, (2, k), device=DEV, generator=g))


def _rmat(n, m, g):
    """m distinct pairs of the recursive matrix over n = 2^scale vertices, ids permuted."""
    a, b, c = _RMAT_ABC
    perm = torch.randperm(n, device=DEV, generator=g)

    def draw_pairs(total):
        us, vs = [], []
        for at in range(0, total, 1 << 24):
            k = min(total - at, 1 << 24)
            u = torch.zeros(k, dtype=torch.int64, device=DEV)
            v = torch.zeros_like(u)
            for _ in range(n.bit_length() - 1):
                r = torch.rand(k, device=DEV, generator=g)
                ub = r >= a + b
                vb = ((r >= a) & ~ub) | (r >= a + b + c)
                u = 2 * u + ub
                v = 2 * v + vb
            us.append(perm[u])
            vs.append(perm[v])
        return torch.cat(us), torch.cat(vs)

    return _distinct(n, m, g, draw_pairs)


def _debruijn(n, m, g, k=21):
    """n distinct 21-mers of a random sequence with short tandem repeats (the graph's few triangles)
    and of mutated copies of its segments; an edge joins k-mers that overlap by k - 1 bases (m of these edges)."""
    bases = int(n / 1.25)
    seq = torch.randint(4, (bases,), dtype=torch.int64, device=DEV, generator=g)
    motifs = torch.randint(4, (bases // 5000, 3), device=DEV, generator=g).repeat(1, 20)  # period-3 tandem repeats
    seq[torch.arange(motifs.shape[0], device=DEV)[:, None] * 5000 + torch.arange(60, device=DEV)] = motifs
    seg = min(10_000, bases // 20)
    copies = bases // (2 * seg)
    at = torch.randint(bases - seg, (copies, 1), device=DEV, generator=g) + torch.arange(seg, device=DEV)
    mut = torch.rand((copies, seg), device=DEV, generator=g) < 0.05
    seq = torch.cat([seq, torch.where(mut, torch.randint(4, (copies, seg), device=DEV, generator=g), seq[at]).reshape(-1)])
    words = torch.zeros(seq.numel() - k + 1, dtype=torch.int64, device=DEV)
    for j in range(k):
        words = words * 4 + seq[j:j + words.numel()]
    words = _exactly(torch.unique(words), n, g).sort().values
    a, b = [], []
    for base in range(4):
        nxt = (words * 4 + base) & ((1 << (2 * k)) - 1)
        to = torch.searchsorted(words, nxt).clamp_(max=n - 1)
        hit = (words[to] == nxt).nonzero().squeeze(1)
        a.append(hit)
        b.append(to[hit])
    return _csr(n, _exactly(_pairs(n, torch.cat(a), torch.cat(b)), m, g))


def _mix_sizes(case):
    """(kind, n, m) per member: sizes and degrees spread evenly over their logarithms, in mixed order."""
    got, k = [], case["count"]
    for i in range(k):
        n = int(case["n_lo"] * (case["n_hi"] / case["n_lo"]) ** ((i + 0.5) / k))
        m = int(n * 4.0 * 16.0 ** ((i * 0.618034) % 1.0) / 2)
        got.append(("rmat", 1 << round(math.log2(n)), m) if i % 2 else ("er", n, m))
    return [got[(i * 7) % k] for i in range(k)] if k % 7 else got


def _graphs(case, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    make = {"er": _er, "rmat": _rmat, "dbg": _debruijn}
    if case["graph"] == "mix":
        return [make[kind](n, m, g) for kind, n, m in _mix_sizes(case)]
    return [make[case["graph"]](case["n"], case["m"], g)]


def _mtx_pairs(off, nbr):
    """The lower triangle's entries (i > j), row by row."""
    rows = torch.repeat_interleave(torch.arange(off.numel() - 1, device=DEV), off[1:] - off[:-1])
    low = rows > nbr
    return rows[low], nbr[low]


def _mtx_text(off, nbr):
    i, j = _mtx_pairs(off, nbr)
    n = off.numel() - 1
    digits = len(str(n))
    cols = torch.full((i.numel(), 2 * digits + 2), ord(" "), dtype=torch.uint8, device=DEV)
    show = torch.ones_like(cols, dtype=torch.bool)
    for at, v in ((0, i + 1), (digits + 1, j + 1)):
        for d in range(digits):
            p = 10 ** (digits - 1 - d)
            cols[:, at + d] = (v // p % 10 + ord("0")).to(torch.uint8)
            show[:, at + d] = v >= p
    cols[:, -1] = ord("\n")
    head = f"%%MatrixMarket matrix coordinate pattern symmetric\n{n} {n} {i.numel()}\n".encode()
    return head + cols[show].cpu().numpy().tobytes()


def _host(off, nbr, ids):
    return off.cpu().numpy().astype(np.uint64), nbr.cpu().numpy().astype(ids)


def prepare(case, seed):
    graphs, op = _graphs(case, seed), case["op"]
    state = {"op": op}
    if op == "pkt":
        off, nbr = graphs[0]
        state["off"], state["nbr"] = off, nbr.to(torch.int32)
        state["out"] = torch.empty_like(state["nbr"])
        state["opts"] = pkt.PktOptions(out_bits=32)
    elif op == "batch":
        state["graphs"] = [_host(o, v, np.uint32) for o, v in graphs]
        state["opts"] = pkt.PktOptions(out_bits=32)
    elif op == "mtx":
        state["text"] = _mtx_text(*graphs[0])
    else:
        state["off"], state["nbr"] = _host(*graphs[0], np.uint64)
        state["opts"] = pkt.PktOptions(out_bits=case.get("bits", 32))
    return state


def run(state):
    op = state["op"]
    if op == "pkt":
        off, nbr, out = state["off"], state["nbr"], state["out"]
        pkt.run_pkt_device(off.data_ptr(), off.numel(), nbr.data_ptr(), nbr.numel(), out.data_ptr(), state["opts"])
        return out
    if op == "batch":
        return [truss for truss, _, _ in pkt.run_batch(state["graphs"], state["opts"])]
    if op == "mtx":
        off, nbr = pkt.mtx_to_csr(state["text"])
        return {"offsets": off, "neighbours": nbr}
    off, nbr, opts = state["off"], state["nbr"], state["opts"]
    if op == "pkt_host":
        return pkt.run_pkt(off, nbr, opts)[0]
    if op == "triangles":
        return pkt.run_triangles(off, nbr, opts)[0]
    if op == "kcore":
        return pkt.run_kcore(off, nbr, opts)[0]
    local, transitivity, average, _ = pkt.run_clustering(off, nbr, opts)
    return {"local": local, "transitivity": transitivity, "average": average}


# ---- work --------------------------------------------------------------------------------


def work(case):
    """Bytes of the inputs read once and the results written once; a graph algorithm's comparisons are not counted."""
    op = case["op"]
    if case["graph"] == "mix":
        n, w = (sum(s[k] for s in _mix_sizes(case)) * k for k in (1, 2))
    else:
        n, w = case["n"], 2 * case["m"]
    ids, out = {"pkt": (4, 4 * w), "batch": (4, 4 * w), "pkt_host": (8, case.get("bits", 32) // 8 * w),
                "triangles": (8, 4 * w), "kcore": (8, 4 * n), "clustering": (8, 8 * n), "mtx": (0, 8 * (n + w))}[op]
    text = w * math.log10(10 * n) if op == "mtx" else 8 * n  # two numbers and their separators per entry
    return {"bytes": text + ids * w + out, "flops": 0}


# ---- the same results by plain torch -----------------------------------------------------


def _triangles(off, nbr, keep):
    """Undirected edge id per slot, triangles per edge and, with `keep`, each triangle's three edge ids."""
    n = off.numel() - 1
    deg = off[1:] - off[:-1]
    src = torch.repeat_interleave(torch.arange(n, device=DEV), deg)
    rank = deg * n + torch.arange(n, device=DEV)
    out = rank[src] < rank[nbr]
    a, b = src[out], nbr[out]
    keys = a * n + b
    eid = torch.searchsorted(keys, torch.where(out, src, nbr) * n + torch.where(out, nbr, src))
    pos = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(torch.bincount(a, minlength=n), 0, out=pos[1:])
    d = pos[1:] - pos[:-1]
    x, y = torch.where(d[a] <= d[b], a, b), torch.where(d[a] <= d[b], b, a)  # the shorter out-list, the longer
    ends = torch.cumsum(d[x], 0)
    sup = torch.zeros(a.numel(), dtype=torch.int64, device=DEV)
    kept, at, m = [], 0, a.numel()
    while at < m:
        base = int(ends[at - 1]) if at else 0
        to = max(at + 1, int(torch.searchsorted(ends, base + (1 << 26), right=True)))
        e = torch.repeat_interleave(torch.arange(at, to, device=DEV), d[x[at:to]])
        f = pos[x[e]] + torch.arange(e.numel(), device=DEV) + base - (ends[e] - d[x[e]])
        want = y[e] * n + b[f]
        h = torch.searchsorted(keys, want).clamp_(max=m - 1)
        hit = keys[h] == want
        three = [t[hit] for t in (e, f, h)]
        for t in three:
            sup += torch.bincount(t, minlength=m)
        if keep:
            kept.append([t.to(torch.int32) for t in three])
        at = to
    return eid, sup, [torch.cat([k[i] for k in kept]).long() for i in range(3)] if kept else None


def _truss(off, nbr):
    eid, sup, tri = _triangles(off, nbr, True)
    sup, level = sup.clone(), torch.zeros_like(sup)
    alive, k = torch.ones_like(sup, dtype=torch.bool), 0
    while bool(alive.any()):
        front = alive & (sup <= k)
        if not bool(front.any()):
            k = int(sup[alive].min())
            continue
        level[front] = k
        alive &= ~front
        if tri is not None:
            gone = front[tri[0]] | front[tri[1]] | front[tri[2]]
            for t in tri:
                sup -= torch.bincount(t[gone], minlength=sup.numel())
            tri = [t[~gone] for t in tri]
    return level[eid] + 2


def _cores(off, nbr):
    n = off.numel() - 1
    deg = off[1:] - off[:-1]
    core, alive, k = torch.zeros_like(deg), deg > 0, 1
    src = torch.repeat_interleave(torch.arange(n, device=DEV), deg)
    dst, deg = nbr, deg.clone()
    while bool(alive.any()):
        front = alive & (deg <= k)
        if not bool(front.any()):
            k = int(deg[alive].min())
            continue
        core[front] = k
        alive &= ~front
        deg -= torch.bincount(dst[front[src]], minlength=n)
        left = alive[src] & alive[dst]
        src, dst = src[left], dst[left]
    return core


def exact(case, seed):
    op = case["op"]
    if op in ("pkt", "pkt_host", "batch") and (op == "batch" or case["graph"] == "rmat" and case["n"] > 1 << 16):
        return None  # the plain peel would take minutes
    graphs = _graphs(case, seed)
    off, nbr = graphs[0]
    n = off.numel() - 1
    if op in ("pkt", "pkt_host"):
        truss = _truss(off, nbr)
        return truss.to(torch.int32) if op == "pkt" else truss.cpu().numpy().astype("u1" if case["bits"] == 8 else "u4")
    if op == "kcore":
        return _cores(off, nbr).cpu().numpy().astype(np.uint32)
    if op == "mtx":
        return dict(zip(("offsets", "neighbours"), _host(off, nbr, np.uint64)))
    eid, sup, _ = _triangles(off, nbr, False)
    if op == "triangles":
        return sup[eid].cpu().numpy().astype(np.uint32)
    deg = (off[1:] - off[:-1]).double()
    src = torch.repeat_interleave(torch.arange(n, device=DEV), off[1:] - off[:-1])
    tri = torch.zeros(n, dtype=torch.int64, device=DEV).index_add_(0, src, sup[eid])
    possible = deg * (deg - 1) / 2
    local = torch.where(possible > 0, ((tri + 1) // 2).double() / possible.clamp(min=1), torch.zeros_like(deg))
    return {"local": local.cpu().numpy(), "transitivity": int(tri.sum()) // 3 / 2.0 / float(possible.sum()),
            "average": float(local.sum()) / n}
