"""Calls on a stream that is not torch's current one: the memory they use is theirs
until that stream is done with it.

The lifetime tests launch nothing: the library's entry point is replaced by one that
notes its pointers, and the caching allocator is asked for the same sizes again while
the launch stream is held back.
"""
import numpy as np
import pytest
import torch

from gputrianglecounting_b200 import _lib, api, graphs, serve
from oracle import oracle

pytestmark = pytest.mark.gpu

HOLD = 1_000_000_000                    # clock cycles a stream is held back, half a second


class Noting:
    """The library, but for one entry point, which notes its arguments and launches nothing."""

    def __init__(self, name):
        self._lib, self._name, self.args = _lib.load(), name, None

    def __getattr__(self, name):
        if name != self._name:
            return getattr(self._lib, name)

        def note(*args):
            self.args = args
            return 0
        return note


def held_stream(cuda):
    s = torch.cuda.Stream(cuda)
    with torch.cuda.stream(s):
        torch.cuda._sleep(HOLD)
    return s


def handed_out_again(sizes, cuda):
    """Pointers that the current stream's next allocations of these sizes get."""
    tensors = [torch.empty(size, dtype=torch.uint8, device=cuda) for size in sizes for _ in range(4)]
    return {t.data_ptr() for t in tensors}


def test_subset_memory_outlives_the_call(cuda, monkeypatch):
    g = graphs.erdos_renyi(60000, 8.0, 5, cuda)
    v = torch.arange(80000, device=cuda, dtype=torch.int32)[::2] % g.n       # 40,000 vertices
    v = torch.stack([v, v], 1)[:, 0]                                         # not contiguous
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    lib = Noting("gtc_count_subset_ws")
    monkeypatch.setattr(api._lib, "load", lambda: lib)
    s = held_stream(cuda)
    out = api.count_subset(g.off, g.ind, v, stream=s)
    ws, ws_bytes = lib.args[8], lib.args[9]
    vertices, count = lib.args[5], lib.args[6]
    assert lib.args[7] == out.data_ptr() and count == 40000
    del out
    again = handed_out_again([ws_bytes, 4 * count, 8 * count], cuda)
    assert not s.query(), "the stream was not held back"
    assert ws not in again and vertices not in again and lib.args[7] not in again


def test_subset_on_a_side_stream(cuda):
    """The current stream allocates and overwrites memory of the same sizes meanwhile, and is
    itself behind when the call is made."""
    g = graphs.rmat(16, 8, 3, device=cuda)
    v = torch.randperm(g.n, device=cuda, generator=torch.Generator(cuda).manual_seed(1))
    v = torch.stack([v[:40000].to(torch.int32)] * 2, 1)[:, 0]
    r, _, _, _ = oracle.per_vertex(g.off.cpu().numpy(), g.ind.cpu().numpy())
    want = r[v.cpu().numpy()]
    size = api.TriangleCounter(cuda).workspace_bytes(g.n, g.nnz, 64) + 256
    torch.cuda.synchronize()
    s = torch.cuda.Stream(cuda)
    torch.cuda._sleep(HOLD)
    outs = []
    for _ in range(4):
        outs.append(api.count_subset(g.off, g.ind, v, stream=s))
        junk = [torch.full((k,), 0x5a, dtype=torch.uint8, device=cuda)
                for k in (size, 4 * v.numel(), 8 * v.numel())]
        del junk
    s.synchronize()
    for out in outs:
        assert np.array_equal(out.cpu().numpy(), want)


def test_one_shot_count_memory_outlives_the_call(cuda, monkeypatch):
    g = graphs.erdos_renyi(60000, 8.0, 5, cuda)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    lib = Noting("gtc_count_tuned")
    monkeypatch.setattr(api._lib, "load", lambda: lib)
    s = held_stream(cuda)
    out = api.count_triangles(g.off, g.ind, stream=s)
    r, t, lcc, total, ws, ws_bytes = lib.args[6:12]
    assert r == out.r.data_ptr() and total == out.global_counts.data_ptr()
    del out
    again = handed_out_again([ws_bytes, 8 * g.n, 24], cuda)
    assert not s.query(), "the stream was not held back"
    assert not {r, t, lcc, total, ws} & again


def test_counter_workspace_dropped_while_another_stream_uses_it(cuda, monkeypatch):
    """A workspace allocated on the current stream, used on s, then outgrown."""
    a, b = graphs.erdos_renyi(60000, 8.0, 5, cuda), graphs.erdos_renyi(90000, 8.0, 5, cuda)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    lib = Noting("gtc_count_tuned")
    monkeypatch.setattr(api._lib, "load", lambda: lib)
    counter = api.TriangleCounter(cuda)
    counter.count(a.off, a.ind, mode="oriented")
    s = held_stream(cuda)
    counter.count(a.off, a.ind, mode="oriented", stream=s)
    ws, ws_bytes = lib.args[10], lib.args[11]
    counter.count(b.off, b.ind, mode="oriented")
    assert lib.args[10] != ws
    again = handed_out_again([ws_bytes], cuda)
    assert not s.query(), "the stream was not held back"
    assert ws not in again


def test_one_shot_count_on_a_side_stream(cuda):
    g = graphs.rmat(14, 8, 3, device=cuda)
    r, t, _, _ = oracle.per_vertex(g.off.cpu().numpy(), g.ind.cpu().numpy())
    size = api.TriangleCounter(cuda).workspace_bytes(g.n, g.nnz, 64)
    torch.cuda.synchronize()
    s = torch.cuda.Stream(cuda)
    torch.cuda._sleep(HOLD)
    outs = []
    for _ in range(4):
        outs.append(api.count_triangles(g.off, g.ind, stream=s))
        assert api.validate_csr(g.off, g.ind, stream=s)[0] == 0
        junk = [torch.full((k,), 0x5a, dtype=torch.uint8, device=cuda) for k in (size, 8 * g.n, 256)]
        del junk
    s.synchronize()
    for out in outs:
        assert np.array_equal(out.r.cpu().numpy(), r) and np.array_equal(out.t.cpu().numpy(), t)


def test_batch_memory_outlives_the_call(cuda, monkeypatch):
    gs = [graphs.erdos_renyi(20000, 8.0, k, cuda) for k in range(3)]
    batch = graphs.concat_graphs(gs, cuda)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    lib = Noting("gtc_count_batch")
    monkeypatch.setattr(api._lib, "load", lambda: lib)
    s = held_stream(cuda)
    out = api.BatchCounter(cuda).count(batch, stream=s)
    r, _, lcc, total, ws, ws_bytes = lib.args[6:12]
    assert r == out.r.data_ptr() and total == out.graph_T.data_ptr()
    del out
    again = handed_out_again([ws_bytes, 8 * batch.total_n, 24], cuda)
    assert not s.query(), "the stream was not held back"
    assert not {r, lcc, total, ws} & again


def test_packs_in_flight_keep_their_staging(cuda):
    """Packs on a stream that is held back, by one counter and by counters that are dropped at
    once: each copies the graphs that it was given."""
    gs = [graphs.erdos_renyi(3000 + 100 * k, 6.0, k, cuda) for k in range(6)]
    torch.cuda.synchronize()
    counter = api.BatchCounter(cuda)
    s = held_stream(cuda)
    one = [counter.pack(gs[k:k + 2], stream=s) for k in (0, 2, 4)]
    other = [api.BatchCounter(cuda).pack(gs[k:k + 2], stream=s) for k in (0, 2, 4)]
    s.synchronize()
    for k, a, b in zip((0, 2, 4), one, other):
        want = graphs.concat_graphs(gs[k:k + 2], cuda)
        for got in (a, b):
            assert torch.equal(got.vstart, want.vstart) and torch.equal(got.off, want.off)
            assert torch.equal(got.ind, want.ind)


def test_served_results_are_copied_before_the_slot_is_reused(cuda):
    """The copies of a finished batch's r wait on a held-back stream while the slot's stream
    allocates and overwrites memory of the same size."""
    gs = [graphs.erdos_renyi(20000, 8.0, k, cuda) for k in range(3)]
    server = serve.CountServer(gs, cuda, slots=1, keep_vertex_results=True)
    slot = server.slots[0]
    reqs = [serve.Request(k, k, 0.0, g.n, g.nnz) for k, g in enumerate(gs)]
    torch.cuda.synchronize()
    assert server._launch(slot, reqs)
    slot.stream.synchronize()
    want, size = slot.out.r.clone(), 8 * slot.out.r.numel()
    torch.full((size,), 0, dtype=torch.uint8, device=cuda)     # its kernel is loaded now
    torch.cuda.synchronize()

    def held(*args, _of=torch.Tensor.clone):      # the host has T, the copies are yet to run
        torch.cuda._sleep(HOLD)
        return _of(*args)
    with pytest.MonkeyPatch.context() as patch:
        patch.setattr(torch.Tensor, "clone", held)
        server._finish(slot, 0.0)
    with torch.cuda.stream(slot.stream):
        junk = [torch.full((size,), 0x5a, dtype=torch.uint8, device=cuda) for _ in range(8)]
    torch.cuda.synchronize()
    del junk
    assert torch.equal(torch.cat([q.r for q in reqs]), want)
