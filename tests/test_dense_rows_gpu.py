"""Rows with long lists outside a core, looked up in a table or in a bitmap: list lengths on both
sides of the line between them, rows of more members than either holds at a time, the largest
graph that a bitmap spans, and graphs whose lists also name core positions.  Compared exactly, with
the oracle or with the closed form of the graph."""
import numpy as np
import pytest
import torch

from gputrianglecounting_b200 import api, graphs as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _ring(n, k, dev):
    """Vertex i joined to i +- 1 .. k: 3 k (k - 1) / 2 triangles through every vertex."""
    i = torch.arange(n, device=dev).repeat_interleave(k)
    return G.csr_from_pairs(i, (i + torch.arange(1, k + 1, device=dev).repeat(n)) % n, n)


def _check(g, r, dev):
    counter = api.TriangleCounter(dev)
    want = torch.as_tensor(r).to(dev)
    for tuning in (None, {"labels": 1}, {"labels": 2}):
        res = counter.count(g.off, g.ind, tuning=tuning)
        assert torch.equal(res.r, want) and res.total == int(want.sum()), tuning
        res = counter.count(g.off, g.ind, mode="oriented", tuning=tuning)
        assert res.total == int(want.sum()), tuning


@pytest.mark.parametrize("k", [128, 129, 256, 257, 1024, 1025])
def test_list_lengths(k, cuda):
    g = _ring(4 * k + 41000, k, cuda)
    _check(g, np.full(g.n, 3 * k * (k - 1)), cuda)


@pytest.mark.parametrize("n", [32767, 32768, 32769])
@pytest.mark.parametrize("k", [256, 257, 384, 385])
def test_list_lengths_of_smaller_graphs(k, n, cuda):
    _check(_ring(n, k, cuda), np.full(n, 3 * k * (k - 1)), cuda)


@pytest.mark.parametrize("n", [131071, 131072, 131073])
def test_largest_bitmap(n, cuda):
    g = _ring(n, 520, cuda)
    _check(g, np.full(n, 3 * 520 * 519), cuda)


@pytest.mark.parametrize("clique", [4096, 4097, 4098, 8194])
def test_more_members_than_a_bitmap_counts(clique, cuda):
    """A clique beside a small one, in a batch, whose core is too small for it."""
    i, j = torch.triu_indices(clique, clique, 1, device=cuda)
    g, small = G.csr_from_pairs(i, j, clique), G.complete(20).to(cuda)
    res = api.BatchCounter(cuda).count(G.concat_graphs([small, g, small], cuda))
    per = [(19 * 18, 20), ((clique - 1) * (clique - 2), clique), (19 * 18, 20)]
    want = torch.cat([torch.full((n,), r, device=cuda) for r, n in per])
    assert torch.equal(res.r, want)
    assert res.graph_T.tolist() == [r * n // 6 for r, n in per]


@pytest.mark.parametrize("n", [6000, 7000])
def test_lists_that_name_core_positions(n, cuda):
    """Half the vertices in a dense part, too many for the core, which takes the hubs and leaves
    the others' lists with both kinds of names."""
    rng = np.random.default_rng(n)
    m = n // 2
    a, b = rng.integers(0, m, (2, m * 700))
    hub = np.repeat(np.arange(40), m)
    ends = np.concatenate([b, np.tile(np.arange(m), 40)])
    ids = rng.permutation(n)
    g = G.csr_from_pairs(torch.as_tensor(ids[np.concatenate([a, hub])]),
                         torch.as_tensor(ids[ends]), n).numpy()
    r = O.per_vertex(g.off, g.ind)[0]
    _check(G.CSRGraph(torch.as_tensor(g.off).to(cuda), torch.as_tensor(g.ind).to(cuda)), r, cuda)
