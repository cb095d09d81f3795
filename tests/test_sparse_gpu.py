"""Large uniform graphs of mean degree up to 4, whose rows' pairs are looked up one by one: at the
line, with rows of every length that is not a block's, and with longer ones.  Compared exactly."""
import numpy as np
import pytest
import torch

from gputrianglecounting_b200 import api, graphs as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu

N = 1 << 18                             # vertices from which on sparse graphs go this way


def _check(g, dev):
    r, t, lcc, total = O.per_vertex(g.off, g.ind)
    off, ind = torch.as_tensor(g.off).to(dev), torch.as_tensor(g.ind).to(dev)
    counter = api.TriangleCounter(dev)
    for o in (off, off.to(torch.int32)):
        for tuning in (None, {"labels": 1}, {"labels": 2}):
            res = counter.count(o, ind, tuning=tuning)
            assert np.array_equal(res.r.cpu().numpy(), r), tuning
            assert np.array_equal(res.lcc.cpu().numpy().view(np.int64), lcc.view(np.int64))
            assert res.total == total
            assert counter.count(o, ind, mode="oriented", tuning=tuning).total == total
    return total


def _cliques(n, size, more=()):
    """Cliques of `size` on every (size^2 / 4 + 1)th vertices of n, and more pairs."""
    i, j = np.triu_indices(size, 1)
    at = np.arange(0, n - size, max(size, size * size // 3))[:, None]
    a, b = (at + i).ravel(), (at + j).ravel()
    for x, y in more:
        a, b = np.concatenate([a, x]), np.concatenate([b, y])
    return G.csr_from_pairs(torch.as_tensor(a), torch.as_tensor(b), n).numpy()


@pytest.mark.parametrize("n", [N - 1, N, N + 31, N + 33])
@pytest.mark.parametrize("degree", [0.01, 2.0, 3.9, 4.1])
def test_random(n, degree, cuda):
    _check(G.erdos_renyi(n, degree, 5).numpy(), cuda)


@pytest.mark.parametrize("size", [3, 4, 8, 9, 16, 24])
def test_cliques(size, cuda):
    """Rows of 2 .. 23 members, all of whose pairs are edges."""
    assert _check(_cliques(N + 5, size), cuda) > 0


@pytest.mark.parametrize("size", [62, 64, 65, 66, 80])
def test_cliques_of_wide_rows(size, cuda):
    """Cliques around the longest row that is not wide; the larger ones' degrees make the graph
    skewed, and it takes the general path."""
    assert _check(_cliques(N + 5, size), cuda) > 0


def test_geometric(cuda):
    assert _check(G.rgg2d(N + 77, 3.5, 4).numpy(), cuda) > 0


def test_no_edges(cuda):
    assert _check(G.csr_from_pairs(torch.zeros(0, dtype=torch.int64),
                                   torch.zeros(0, dtype=torch.int64), N + 1).numpy(), cuda) == 0


def test_ids_out_of_range(cuda):
    g = _cliques(N, 5)
    bad = np.array(g.ind, np.int32)
    t = O.per_vertex(g.off, g.ind)[1]
    # the last entry of the last rows points outside: their triangles go, the others' stay
    rows = np.flatnonzero(np.diff(g.off))[-5:]
    bad[g.off[rows + 1] - 1] = N + 9
    counter = api.TriangleCounter(cuda)
    res = counter.count(torch.as_tensor(g.off).to(cuda), torch.as_tensor(bad).to(cuda))
    keep = np.setdiff1d(np.arange(N), rows)
    assert np.array_equal(res.t.cpu().numpy()[keep], t[keep])
    with pytest.raises(api.GTCError):
        counter.check_status()
