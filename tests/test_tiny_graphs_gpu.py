"""Batches of many tiny graphs, of which a block chooses several cores.  Compared exactly."""
import numpy as np
import pytest

from gputrianglecounting_b200 import api, graphs as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1184, 4735, 4736, 9471, 9472, 14300])
def test_batch_of_tiny_graphs(count, cuda):
    """Graphs of 0 to 70 vertices, the largest without long rows, some all core and some with a
    hub, in batches of one, two and three graphs per block."""
    rng = np.random.default_rng(count)
    kinds = [G.complete(n) for n in (1, 2, 3, 20, 63, 64, 65, 66, 70)]
    kinds += [G.star(n) for n in (5, 64, 65, 66, 67, 200)] + [G.wheel(80), G.cycle(9)]
    kinds += [G.erdos_renyi(n, 6, n) for n in (16, 40, 64, 65, 600)]
    kinds += [G.from_edge_list(n, []) for n in (0, 1, 64, 65)]
    kinds = [k.numpy() for k in kinds]
    ref = [O.per_vertex(k.off, k.ind) if k.n else (np.zeros(0, np.int64),) * 3 + (0,)
           for k in kinds]
    pick = rng.integers(0, len(kinds), count)
    batch = G.concat_graphs([kinds[i] for i in pick], cuda)
    for tuning in (None, {"labels": 1}, {"labels": 2}):
        res = api.BatchCounter(cuda).count(batch, tuning=tuning)
        assert np.array_equal(res.r.cpu().numpy(), np.concatenate([ref[i][0] for i in pick]))
        assert np.array_equal(res.graph_T.cpu().numpy() * 6, np.array([ref[i][3] for i in pick]))
