"""The counting kernels at the sizes where their paths change: rows of core
members around every tile and chunk size, tiles and tables around their list
lengths, signatures, mixed batches, placement of ids out of range, the
vertex-subset rules and the CSR check's chunk edges.  Everything is integer
and exact, so every comparison is with tolerance 0 (lcc: the same division of
the same integers)."""
import ctypes

import numpy as np
import pytest
import torch

from gputrianglecounting_b200 import _lib, api, graphs as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _csr(n, a, b):
    """Simple symmetric CSR of the pairs (a, b), duplicates and loops dropped."""
    return G.csr_from_pairs(torch.as_tensor(np.asarray(a, np.int64)),
                            torch.as_tensor(np.asarray(b, np.int64)), n).numpy()


def _pairs(g):
    row = np.repeat(np.arange(g.n), np.diff(g.off))
    return row, np.asarray(g.ind, np.int64)


def _ring(n, k):
    """Vertex i joined to i +- 1 .. k: a forward list of k, three quarters of
    the pairs closed."""
    i = np.repeat(np.arange(n), k)
    return _csr(n, i, (i + np.tile(np.arange(1, k + 1), n)) % n)


def _count_everywhere(g, dev, tunings=(None, {"labels": 1}, {"labels": 2})):
    """All outputs of a count with either offset type, aligned and not, in
    every launch form, and the global count alone, against the oracle."""
    r, t, lcc, total = O.per_vertex(g.off, g.ind)
    counter = api.TriangleCounter(dev)
    ind = torch.as_tensor(np.asarray(g.ind, np.int32)).to(dev)
    shifted = torch.empty(ind.numel() + 1, dtype=torch.int32, device=dev)
    shifted[1:] = ind
    for bits, d_ind in ((torch.int32, ind), (torch.int64, shifted[1:])):
        d_off = torch.as_tensor(np.asarray(g.off, np.int64)).to(dev, bits)
        for tun in tunings:
            res = counter.count(d_off, d_ind, tuning=tun)
            one = counter.count(d_off, d_ind, mode="oriented", tuning=tun)
            torch.cuda.synchronize()
            assert np.array_equal(res.r.cpu().numpy(), r), tun
            assert np.array_equal(res.t.cpu().numpy(), t), tun
            assert np.array_equal(res.lcc.cpu().numpy().view(np.int64), lcc.view(np.int64)), tun
            assert res.total == total and one.total == total, tun
    counter.check_status()
    return r


def _core_graph(members, hubs, n, seed):
    """`hubs` vertices joined at random (half of their pairs) and, for every
    m of members, three vertices with m of them as neighbours."""
    rng = np.random.default_rng(seed)
    i, j = np.triu_indices(hubs, 1)
    pick = rng.random(i.size) < 0.5
    a, b = [i[pick]], [j[pick]]
    for k, m in enumerate(np.repeat(members, 3)):
        a.append(np.full(m, hubs + k))
        b.append(rng.choice(hubs, m, replace=False))
    a, b = np.concatenate(a), np.concatenate(b)
    ids = rng.permutation(n)                      # hubs anywhere among the ids
    return _csr(n, ids[a], ids[b])


@pytest.mark.parametrize("n", [16384, 300000])
@pytest.mark.parametrize("members,hubs", [
    ([1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65], 400),
    ([127, 128, 129, 255, 256, 257, 511, 512, 513], 700),
    ([1023, 1024, 1025, 1056, 1290], 1300),       # more than one chunk of members
])
def test_core_rows(members, hubs, n, cuda):
    _count_everywhere(_core_graph(members, hubs, n, hubs), cuda)


@pytest.mark.parametrize("n,k", [(40, 1), (1000, 2), (5003, 7), (5003, 31), (5003, 32),
                                 (5003, 33), (20011, 64), (20011, 65), (20011, 128),
                                 (20011, 129), (262144, 5)])
def test_ring_rows(n, k, cuda):
    """Uniform graphs: tiles whose rows share nearly all members (lists of up
    to 32, one stream) and tables (rows of more than 64 entries)."""
    r = _count_everywhere(_ring(n, k), cuda)
    assert k == 1 or (r == 3 * k * (k - 1)).all()


@pytest.mark.parametrize("length", [1, 31, 32, 33, 63, 64])
def test_tile_lists(length, cuda):
    """Short rows all of whose neighbours have higher ids, so that lists are
    as long as the rows: runs of a ring in the upper half, no two rows' runs
    alike, so a tile's members are mostly distinct (more than 96)."""
    n = 6000
    rng = np.random.default_rng(length)
    low = np.repeat(np.arange(n // 2), length)
    run = np.repeat(rng.integers(0, n // 2, n // 2), length) + np.tile(np.arange(length), n // 2)
    row, col = _pairs(_ring(n // 2, 2))
    _count_everywhere(_csr(n, np.concatenate([low, row + n // 2]),
                           np.concatenate([run % (n // 2) + n // 2, col + n // 2])), cuda)


def _sparse_er(n, degree, seed):
    """An Erdos-Renyi graph with triangles: a hundred ids joined in runs."""
    row, col = _pairs(G.erdos_renyi(n, degree, seed).numpy())
    x = np.random.default_rng(seed).choice(n, 100, replace=False)
    return _csr(n, np.concatenate([row, x[:-1], x[:-2]]),
                np.concatenate([col, x[1:], x[2:]]))


@pytest.mark.parametrize("n,degree", [(32767, 12), (32768, 8.1), (40001, 12), (33000, 24),
                                      (33000, 45), (262147, 9)])
def test_signatures(n, degree, cuda):
    """Sparse uniform graphs of the smallest call with signatures up (and one
    below), lists of up to 8, 16, 32 and 64 members and longer ones; with a
    star beside it, the graph is not uniform and takes the general path, to
    the same counts."""
    g = _sparse_er(n, degree, 7)
    r = _count_everywhere(g, cuda)
    assert r.max() > 0
    row, col = _pairs(g)
    hub, leaves = n, np.arange(n + 1, n + 1 + 8 * int(degree) + 65)
    both = _csr(n + 1 + leaves.size, np.concatenate([row, np.full(leaves.size, hub)]),
                np.concatenate([col, leaves]))
    res = api.TriangleCounter(cuda).count(torch.as_tensor(both.off).to(cuda),
                                          torch.as_tensor(np.asarray(both.ind, np.int32)).to(cuda))
    torch.cuda.synchronize()
    assert np.array_equal(res.r.cpu().numpy()[:n], r)


@pytest.mark.parametrize("clique", [8, 129, 1025, 1026, 1500])
def test_mixed_batch(clique, cuda):
    """One batch of graphs that take different paths: signatures, tiles, a
    core, all core, and cliques too large for their core (tables of 1,024
    members at a time)."""
    n = max(clique + 75, 800)
    i, j = np.triu_indices(clique, 1)
    gs = [G.from_edge_list(3, [(0, 1), (1, 2), (0, 2)]).numpy(), _csr(n, i, j + n - clique),
          _sparse_er(40001, 12, 3), _ring(700, 30), _csr(n, i, j), G.rmat(13, 16, 5).numpy(),
          G.complete(200).numpy(), G.erdos_renyi(600, 5, 1).numpy(), _sparse_er(601, 10, 2),
          G.rgg2d(9000, 14, 2).numpy(), G.from_edge_list(0, []).numpy()]
    batch = G.concat_graphs(gs, cuda)
    vstart = batch.vstart.cpu().numpy()
    for tun in (None, {"labels": 1}, {"labels": 2}):
        res = api.BatchCounter(cuda).count(batch, tuning=tun)
        torch.cuda.synchronize()
        for k, g in enumerate(gs):
            r, _, lcc, total = O.per_vertex(g.off, g.ind)
            sl = slice(vstart[k], vstart[k + 1])
            assert np.array_equal(res.r.cpu().numpy()[sl], r), (tun, k)
            assert np.array_equal(res.lcc.cpu().numpy()[sl].view(np.int64),
                                  lcc.view(np.int64)), (tun, k)
            assert int(res.graph_T[k]) * 6 == total, (tun, k)


@pytest.mark.parametrize("make", [lambda: _ring(3000, 12), lambda: _sparse_er(40001, 12, 5),
                                  lambda: _core_graph([40, 70], 300, 8192, 1)])
def test_ids_out_of_range_are_skipped(make, cuda):
    """Ids below 0 and from n on, first and last in their rows, change nothing
    but the status."""
    g = make()
    rng = np.random.default_rng(1)
    bad = set(rng.choice(g.n, 200, replace=False).tolist())
    rows = np.split(np.asarray(g.ind, np.int32), g.off[1:-1])
    rows = [np.concatenate([[-5], x, [g.n, 2 ** 31 - 1]]) if v in bad else x
            for v, x in enumerate(rows)]
    off = np.concatenate([[0], np.cumsum([x.size for x in rows])])
    counter = api.TriangleCounter(cuda)
    t = O.per_vertex(g.off, g.ind)[1]
    for labels in (0, 1, 2):
        res = counter.count(torch.as_tensor(off).to(cuda),
                            torch.as_tensor(np.concatenate(rows).astype(np.int32)).to(cuda),
                            tuning={"labels": labels})
        torch.cuda.synchronize()
        assert np.array_equal(res.t.cpu().numpy(), t)
        with pytest.raises(api.GTCError):
            counter.check_status()


@pytest.mark.parametrize("make", [lambda: G.rmat(12, 24, 2).numpy(), lambda: _ring(2000, 40),
                                  lambda: _csr(1600, *np.triu_indices(1500, 1))])
def test_smallest_workspace(make, cuda):
    """The smallest workspace that is accepted, which may hold a smaller core,
    gives the same counts; one byte less is refused."""
    g = make()
    lib = _lib.load()
    off = torch.as_tensor(np.asarray(g.off, np.int64)).to(cuda)
    ind = torch.as_tensor(np.asarray(g.ind, np.int32)).to(cuda)
    r = torch.empty(g.n, dtype=torch.int64, device=cuda)
    full = api.TriangleCounter(cuda).workspace_bytes(g.n, ind.numel(), 64)
    ws = torch.empty(full, dtype=torch.uint8, device=cuda)

    def run(size):
        return lib.gtc_count(off.data_ptr(), 64, ind.data_ptr(), g.n, ind.numel(), 0,
                             r.data_ptr(), None, None, None, ws.data_ptr(), size, None)

    lo, hi = 0, full                              # refused, accepted
    while hi - lo > 1:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if run(mid) == 0 else (mid, hi)
    torch.cuda.synchronize()
    r.zero_()
    torch.cuda.synchronize()
    assert run(lo) != 0
    torch.cuda.synchronize()
    assert not r.any()
    assert run(hi) == 0
    torch.cuda.synchronize()
    assert np.array_equal(r.cpu().numpy(), O.per_vertex(g.off, g.ind)[0])


@pytest.mark.parametrize("which", ["rmat", "ring", "er"])
@pytest.mark.parametrize("count", [1, 31, 1023, 1024, 8191, 8192, 16383, 16384, 40000])
def test_subset_rules(which, count, cuda):
    """A block, a warp per listed vertex or a count of the whole graph, by the
    number of vertices (some listed more than once): the oracle's sums, and
    the same through the entry point that takes no workspace."""
    g = {"rmat": lambda: G.rmat(13, 24, 3).numpy(), "ring": lambda: _ring(9001, 70),
         "er": lambda: G.erdos_renyi(30000, 20, 1).numpy()}[which]()
    v = np.random.default_rng(count).integers(0, g.n, count).astype(np.int32)
    ref = O.subset(g.off, g.ind, v)
    off = torch.as_tensor(np.asarray(g.off, np.int64)).to(cuda)
    ind = torch.as_tensor(np.asarray(g.ind, np.int32)).to(cuda)
    d_v = torch.as_tensor(v).to(cuda)
    assert np.array_equal(api.count_subset(off, ind, d_v).cpu().numpy(), ref)
    out = torch.empty(count, dtype=torch.int64, device=cuda)
    assert _lib.load().gtc_count_subset(off.data_ptr(), 64, ind.data_ptr(), d_v.data_ptr(), count,
                                        out.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), ref)


@pytest.mark.parametrize("n", [255, 256, 257, 512, 1025])
def test_check_at_chunk_edges(n, cuda):
    """The CSR check takes 512 entries per warp: a defect at the first and
    last entry of the array and of a chunk is found, as on the host."""
    g = _ring(n, 1)                               # 2 n entries
    nnz = int(g.off[-1])
    off = torch.as_tensor(np.asarray(g.off, np.int64)).to(cuda)
    for at in sorted({0, 1, 510, 511, 512, 513, nnz // 2, nnz - 1}):
        if at >= nnz:
            continue
        row = int(np.searchsorted(g.off, at, side="right")) - 1
        for value in (int(g.ind[at]), row, n, (row + n // 2) % n):
            ind = np.asarray(g.ind, np.int32).copy()
            ind[at] = value
            code, text = api.validate_csr(off, torch.as_tensor(ind).to(cuda))
            host = G.validate_csr_host(np.asarray(g.off, np.int64), ind)
            assert (code == 0) == (host is None), (at, value, text, host)
