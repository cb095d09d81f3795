"""Cases that stand for what a program does with this counter, at the sizes it meets.

Every case goes through the public entry points of `gputrianglecounting_b200.api`, with the
library's own choice of launch shape unless the case carries a plan that a program would keep.
Graphs are the families the benchmark names: Erdos-Renyi, R-MAT (0.57, 0.19, 0.19, 0.05) and
the Morton-ordered 2D random geometric graph; batches mix Erdos-Renyi and R-MAT graphs.

Operations (`op`):
  count     TriangleCounter.count: r, t, lcc and the global count, or (mode "oriented") the
            global count alone
  call      kernelCall, the reference's operator, int32 or int64
  call_list kernelCall with a vertex list
  subset    count_subset: r of listed vertices
  ingest    validate_csr, then a count: a graph that arrives from outside
  batch     BatchCounter.count of a resident batch
  pack      BatchCounter.pack of separate resident graphs, then the count: a served request batch
"""
from __future__ import annotations

import math

import torch

from gputrianglecounting_b200 import api, graphs

ABCD = (0.57, 0.19, 0.19, 0.05)


def listed():
    return [
        # the smallest calls: launches, allocation and host work dominate (the smoke test's size)
        dict(name="count_rmat10", op="count", family="rmat", scale=10, degree=16.0, bits=32,
             mode="plain"),
        # a small mesh-like graph, the benchmark's ER configuration
        dict(name="count_er16k", op="count", family="er", n=16384, degree=16.0, bits=32,
             mode="plain"),
        # the reference's operator as its callers bind to it, on a mid-sized social-like graph
        dict(name="call_rmat17_i64", op="call", family="rmat", scale=17, degree=24.0, bits=64),
        # the headline workload
        dict(name="count_rmat20", op="count", family="rmat", scale=20, degree=32.0, bits=32,
             mode="plain"),
        # the largest single graph that the server is given
        dict(name="count_rmat22", op="count", family="rmat", scale=22, degree=32.0, bits=64,
             mode="plain"),
        # the benchmark's geometric graph: low degree, local ids
        dict(name="count_rgg4m", op="count", family="rgg", n=4194304, degree=12.0, bits=32,
             mode="plain"),
        # global triangle count only, a sparse skewed graph
        dict(name="oriented_rmat20_ef8", op="count", family="rmat", scale=20, degree=16.0, bits=64,
             mode="oriented"),
        # a large uniform graph of odd size, denser than a mesh
        dict(name="count_er900k_d30", op="count", family="er", n=900001, degree=30.0, bits=64,
             mode="plain"),
        # an eighth of the benchmark's batch with the plan its autotuner picks
        dict(name="batch_512", op="batch", graphs=512, sizes=4, lo=256, hi=262144, tuned=True),
        # one served batch: requests' graphs gathered and counted
        dict(name="pack_64", op="pack", graphs=64, sizes=4, lo=256, hi=262144, tuned=False),
        # clustering of a sample of vertices of the headline graph
        dict(name="subset_rmat20_64k", op="subset", family="rmat", scale=20, degree=32.0, bits=32,
             vertices=65536),
        # a graph from outside: checked, then counted
        dict(name="ingest_rgg1m", op="ingest", family="rgg", n=1000003, degree=14.0, bits=64,
             mode="plain"),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    op = rng.choice(["count", "count", "count", "call", "call_list", "subset", "ingest", "batch",
                     "pack"])
    if op in ("batch", "pack"):
        lo = int(_log_uniform(rng, 64, 4096))
        hi = int(_log_uniform(rng, 2 * lo, 262144))
        most = min(512 if op == "batch" else 128, int(2e7 / (hi / math.log(hi / lo))))
        return dict(op=op, graphs=int(_log_uniform(rng, 2, max(most, 3))),
                    sizes=rng.randint(0, 9999), lo=lo, hi=hi, tuned=rng.random() < 0.5)
    family = rng.choice(["er", "rmat", "rgg"])
    case = dict(op=op, family=family, bits=rng.choice([32, 64]))
    if family == "rmat":
        case["scale"] = rng.randint(8, 18 if op in ("subset", "call_list") else 21)
        case["degree"] = 2.0 * round(rng.uniform(4, 16), 2)
    else:
        # uniform and geometric graphs: at most 48 million adjacency entries
        case["degree"] = round(_log_uniform(rng, 4, 40 if family == "er" else 24), 2)
        case["n"] = int(_log_uniform(rng, 200, min(4e6, 4.8e7 / case["degree"])))
    if op in ("count", "ingest"):
        case["mode"] = rng.choice(["plain", "plain", "oriented"])
    if op in ("subset", "call_list"):
        n = case.get("n") or 1 << case["scale"]
        case["vertices"] = int(_log_uniform(rng, 16, min(n, 65536)))
    return case


def _graph(case, seed, device):
    if case["family"] == "rmat":
        return _rmat(case["scale"], case["degree"], seed, device)
    if case["family"] == "er":
        return graphs.erdos_renyi(case["n"], case["degree"], seed, device)
    return graphs.rgg2d(case["n"], case["degree"], seed, device)


def _rmat(scale, degree, seed, device):
    """2^scale vertices, degree / 2 samples per vertex."""
    g = torch.Generator(device=device)
    g.manual_seed(int(seed))
    src, dst = graphs.rmat_pairs(scale, round(degree * (1 << scale) / 2), ABCD, g, device)
    return graphs.csr_from_pairs(src, dst, 1 << scale)


def _specs(case, seed):
    """The batch's graphs: sizes and kinds belong to the case, the edges to the seed."""
    specs = graphs.batched_specs(case["graphs"], case["sizes"], case["lo"], case["hi"])
    for g, s in enumerate(specs):
        s["seed"] = int(seed) * 1_000_003 + g
    return specs


def _vertices(case, n, seed, device):
    """Listed vertices of a sample: distinct ids in no order."""
    g = torch.Generator(device=device)
    g.manual_seed(int(seed) + 1)
    return torch.randperm(n, generator=g, device=device)[:case["vertices"]]


def prepare(case, seed):
    device = torch.device("cuda", torch.cuda.current_device())
    op = case["op"]
    if op in ("batch", "pack"):
        gs = [graphs.make_spec_graph(s, device) for s in _specs(case, seed)]
        # the shape the autotuner keeps for the benchmark's batch
        tuning = dict(group=16, labels=2, region=4, rows=1, big_chunk=4096,
                      item_len=1024) if case["tuned"] else None
        state = dict(op=op, counter=api.BatchCounter(), tuning=tuning)
        if op == "batch":
            state["batch"] = graphs.concat_graphs(gs, device)
        else:
            state["graphs"] = gs
        return state
    g = _graph(case, seed, device)
    off = g.off.to(torch.int32) if case["bits"] == 32 else g.off
    state = dict(op=op, off=off, ind=g.ind, n=g.n, mode=case.get("mode"))
    if op in ("count", "ingest"):
        state["counter"] = api.TriangleCounter()
        return state
    wide = torch.int64 if case["bits"] == 64 else torch.int32
    if op in ("subset", "call_list"):
        v = _vertices(case, g.n, seed, device)
        state["vertices"] = v.to(torch.int32) if op == "subset" else v.to(wide)
    if op in ("call", "call_list"):
        state["ind"] = g.ind.to(wide)
        state["out"] = torch.zeros(g.n if op == "call" else case["vertices"], dtype=wide,
                                   device=device)
    return state


def run(state):
    op = state["op"]
    if op in ("batch", "pack"):
        batch = state["batch"] if op == "batch" else state["counter"].pack(state["graphs"])
        c = state["counter"].count(batch, tuning=state["tuning"])
        return c.r, c.lcc, c.graph_T
    off, ind = state["off"], state["ind"]
    if op == "subset":
        return api.count_subset(off, ind, state["vertices"])
    if op == "call":
        api.kernelCall(16000, 128, state["n"], off, ind, state["out"], 1, 4, 0)
        return state["out"]
    if op == "call_list":
        v = state["vertices"]
        api.kernelCall(16000, 128, v.numel(), off, ind, state["out"], 1, 4, 0, vertex=v)
        return state["out"]
    reason = api.validate_csr(off, ind)[0] if op == "ingest" else 0
    c = state["counter"].count(off, ind, mode=state["mode"])
    if state["mode"] == "oriented":
        return reason, c.global_counts
    return reason, c.r, c.t, c.lcc, c.global_counts


def _rmat_entries(scale, degree):
    """Expected adjacency entries after duplicates and self-loops are gone."""
    a, b, _, d = ABCD
    samples = degree * (1 << scale) / 2
    pairs = 0.0
    for i in range(scale + 1):
        for m in range(1, scale - i + 1):
            cells = math.comb(scale, i) * math.comb(scale - i, m) * 2.0 ** m
            p = 2 * a ** i * b ** m * d ** (scale - i - m)
            pairs += cells / 2 * -math.expm1(samples * math.log1p(-p))
    return 2 * pairs


def work(case):
    """Every input read once, every output written once; one division per coefficient."""
    op = case["op"]
    if op in ("batch", "pack"):
        specs = _specs(case, 0)
        n = sum(s["n"] for s in specs)
        nnz = sum(s["n"] * s["mean_degree"] if s["kind"] == "er" else
                  _rmat_entries(round(math.log2(s["n"])), 2 * s["edge_factor"]) for s in specs)
        read = 8 * n + 4 * nnz + 8 * len(specs)
        # a pack also writes the batch that it gathers
        return {"bytes": (read if op == "batch" else 2 * read) + 16 * n + 8 * len(specs),
                "flops": n}
    if case["family"] == "rmat":
        n = 1 << case["scale"]
        nnz = _rmat_entries(case["scale"], case["degree"])
    else:
        n, nnz = case["n"], case["n"] * case["degree"]
    word = case["bits"] // 8
    if op in ("call", "call_list"):
        out = word * (n if op == "call" else case["vertices"])
        share = 1.0 if op == "call" else min(1.0, case["vertices"] * (1 + nnz / n) / n)
        return {"bytes": share * (word * (n + 1) + word * nnz) + out, "flops": 0}
    if op == "subset":
        # the listed rows and their neighbours' rows
        share = min(1.0, case["vertices"] * (1 + nnz / n) / n)
        return {"bytes": share * (word * (n + 1) + 4 * nnz) + 12 * case["vertices"], "flops": 0}
    plain = case["mode"] == "plain"
    return {"bytes": word * (n + 1) + 4 * nnz + 24 + (24 * n if plain else 0),
            "flops": n if plain else 0}


_EXACT_PROBES = 3_000_000_000     # most list elements that exact() looks up


def _triangles(off, ind):
    """t(v) of a simple symmetric CSR in plain torch: every edge is turned from its lower to its
    higher end in (degree, id) order, and each element of the shorter forward list of an edge is
    looked up in the other; None where that is too much work."""
    n = off.numel() - 1
    dev = off.device
    deg = off[1:] - off[:-1]
    row = torch.repeat_interleave(torch.arange(n, device=dev), deg)
    col = ind.to(torch.int64)
    up = (deg[col] > deg[row]) | ((deg[col] == deg[row]) & (col > row))
    u, v = row[up], col[up]
    keys = u * n + v                                     # ascending: rows are sorted
    fdeg = torch.bincount(u, minlength=n)
    start = torch.cumsum(fdeg, 0) - fdeg
    t = torch.zeros(n, dtype=torch.int64, device=dev)
    swap = fdeg[u] < fdeg[v]
    a, p = torch.where(swap, v, u), torch.where(swap, u, v)   # look N+(p) up in N+(a)
    k = fdeg[p]
    a, p, k = a[k > 0], p[k > 0], k[k > 0]
    if int(k.sum()) > _EXACT_PROBES:
        return None
    ends = torch.cumsum(k, 0)
    lo, chunk = 0, 1 << 26
    while lo < a.numel():
        base = int(ends[lo - 1]) if lo else 0
        hi = max(lo + 1, int(torch.searchsorted(ends, base + chunk, right=True)))
        kk = k[lo:hi]
        aa, pp = torch.repeat_interleave(a[lo:hi], kk), torch.repeat_interleave(p[lo:hi], kk)
        first = torch.repeat_interleave(start[p[lo:hi]] - (ends[lo:hi] - kk - base), kk)
        w = v[first + torch.arange(first.numel(), device=dev)]
        want = aa * n + w
        at = torch.searchsorted(keys, want).clamp_(max=keys.numel() - 1)
        hit = keys[at] == want
        for end in (aa, pp, w):
            t += torch.bincount(end[hit], minlength=n)
        lo = hi
    return t


def _coefficients(off, t):
    d = (off[1:] - off[:-1]).to(torch.float64)
    pairs = d * (d - 1)
    return torch.where(pairs > 0, 2.0 * t.to(torch.float64) / pairs.clamp(min=1.0),
                       torch.zeros_like(pairs))


def exact(case, seed):
    device = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    op = case["op"]
    if op in ("batch", "pack"):
        rs, ls, ts = [], [], []
        probes = sum(s["n"] * 300 for s in _specs(case, seed))
        if probes > _EXACT_PROBES:
            return None
        for s in _specs(case, seed):
            g = graphs.make_spec_graph(s, device)
            t = _triangles(g.off, g.ind)
            if t is None:
                return None
            rs.append(2 * t)
            ls.append(_coefficients(g.off, t))
            ts.append(t.sum() // 3)
        return torch.cat(rs), torch.cat(ls), torch.stack(ts)
    g = _graph(case, seed, device)
    t = _triangles(g.off, g.ind)
    if t is None:
        return None
    if op in ("subset", "call_list"):
        return 2 * t[_vertices(case, g.n, seed, device)]
    if op == "call":
        return 2 * t
    T = t.sum() // 3
    total = torch.stack([T, 3 * T, 6 * T])
    if case["mode"] == "oriented":
        return 0, total
    return 0, 2 * t, t, _coefficients(g.off, t), total
