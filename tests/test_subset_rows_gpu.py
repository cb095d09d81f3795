"""Vertex subsets whose rows are shared out among blocks: as many long rows as make every team
size, rows that all blocks take beside them, and lists around the sizes at which a block's share
changes.  Whole numbers, compared exactly."""
import numpy as np
import pytest
import torch

from gputrianglecounting_b200 import api, graphs as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _hubs_in_a_dense_graph():
    """3,000 vertices of some 700 neighbours and ten that all others are neighbours of."""
    g = G.erdos_renyi(3000, 700, 3)
    row = torch.repeat_interleave(torch.arange(g.n), g.off[1:] - g.off[:-1])
    hub, all_ = torch.arange(10).repeat_interleave(3000), torch.arange(3000).repeat(10)
    return G.csr_from_pairs(torch.cat([row, hub * 300]), torch.cat([g.ind.long(), all_]), 3000)


@pytest.fixture(scope="module")
def dense():
    g = _hubs_in_a_dense_graph().numpy()
    return g, O.per_vertex(g.off, g.ind)[0]


def _check(g, r, v, dev):
    off, ind = torch.as_tensor(g.off).to(dev), torch.as_tensor(np.asarray(g.ind, np.int32)).to(dev)
    d_v = torch.as_tensor(np.asarray(v, np.int64)).to(dev)
    for o in (off, off.to(torch.int32)):
        assert np.array_equal(api.count_subset(o, ind, d_v.to(torch.int32)).cpu().numpy(), r[v])
    for dtype in (torch.int64, torch.int32):
        out = torch.full((len(v),), -1, dtype=dtype, device=dev)
        api.kernelCall(16000, 128, len(v), off.to(dtype), ind.to(dtype), out, 1, 4, 0,
                       vertex=d_v.to(dtype))
        assert np.array_equal(out.cpu().numpy(), r[v])


@pytest.mark.parametrize("rows", [1, 2, 73, 74, 75, 148, 149, 297, 1023, 1024, 1025, 2990])
@pytest.mark.parametrize("hubs", [0, 1, 10])
def test_long_rows_by_teams(rows, hubs, dense, cuda):
    g, r = dense
    rng = np.random.default_rng(rows)
    some = rng.permutation(np.setdiff1d(np.arange(g.n), np.arange(10) * 300))[:rows]
    v = rng.permutation(np.concatenate([some, np.arange(10)[:hubs] * 300]))
    _check(g, r, v, cuda)


@pytest.mark.parametrize("count", [591, 592, 593, 1184, 1185, 8191, 8192, 16383, 16384, 18944,
                                   18945, 40000])
@pytest.mark.parametrize("kind", ["er", "rgg", "rmat"])
def test_shares_of_a_list(count, kind, cuda):
    """Short rows, rows on both sides of what a warp takes and hubs, in lists around the sizes
    at which the vertices that a block takes grow by one or wrap."""
    g = {"er": lambda: G.erdos_renyi(9001, 40, 1), "rgg": lambda: G.rgg2d(7000, 100, 2),
         "rmat": lambda: G.rmat(13, 16, 3)}[kind]().numpy()
    r = O.per_vertex(g.off, g.ind)[0]
    _check(g, r, np.random.default_rng(count).integers(0, g.n, count), cuda)
