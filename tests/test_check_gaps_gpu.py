"""The CSR check of graphs whose entries lie far apart, with vertices without any between them."""
import numpy as np
import pytest
import torch

from gputrianglecounting_b200 import api, graphs as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gap", [30, 31, 32, 33, 63, 64, 1023, 1024, 1025, 1056, 32768, 33824,
                                 1_100_000])
def test_check_across_gaps(gap, cuda):
    """Triangles with `gap` vertices without entries between them, and the same with one defect."""
    first = np.arange(7) * (gap + 3)
    src = np.concatenate([first, first, first + 1])
    dst = np.concatenate([first + 1, first + 2, first + 2])
    n = int(first[-1]) + 3 + gap
    g = G.csr_from_pairs(torch.as_tensor(src), torch.as_tensor(dst), n).numpy()
    off = torch.as_tensor(np.asarray(g.off, np.int64)).to(cuda)
    ind = np.asarray(g.ind, np.int32)
    assert api.validate_csr(off, torch.as_tensor(ind).to(cuda))[0] == 0
    for at in (0, 5, ind.size // 2, ind.size - 1):
        bad = ind.copy()
        bad[at] = (int(ind[at]) + n // 2) % n
        host = G.validate_csr_host(np.asarray(g.off, np.int64), bad)
        code, text = api.validate_csr(off, torch.as_tensor(bad).to(cuda))
        assert (code == 0) == (host is None), (at, text, host)
