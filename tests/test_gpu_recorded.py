"""Counts recorded from a context's stream and replayed."""
import pytest

import oracle
from bbtc_b200 import Context, Graph, graphs, options

pytestmark = pytest.mark.gpu


def workload(seed):
    g = graphs.rmat(10, 16, seed=seed)
    cuts = graphs.cuts(g, 4, "uni")
    return g, cuts, oracle.count(g.n, g.indptr, g.indices, cuts)


def record(torch, stream, call):
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        call()
    return graph


@pytest.mark.parametrize("kernel", ["auto", "bitmap"])
def test_replayed_counts_keep_apart(kernel):
    """A count recorded from the context's stream and replayed: the graph's next
    wait returns it, other graphs' waits return their own last counts."""
    torch = pytest.importorskip("torch")
    (g, cuts, want_g), (h, hcuts, want_h) = workload(22), workload(23)
    assert want_g != want_h
    o = options(kernel=kernel)
    with Context(0) as ctx:
        a, b = Graph.from_csr(ctx, g, cuts), Graph.from_csr(ctx, h, hcuts)
        stream = torch.cuda.ExternalStream(ctx.stream)
        recorded = []
        try:
            some = a.task_list(sorted=False)[:-1].copy()
            want_some = a.count(some, opts=o)
            assert 0 < want_some < want_g
            assert a.count(opts=o) == want_g and b.count(opts=o) == want_h  # their queues are on the device now
            recorded += [record(torch, stream, lambda: a.count_async(opts=o)),
                         record(torch, stream, lambda: a.count_async(some, opts=o))]
            for graph, want in zip(recorded, (want_g, want_some)):
                with torch.cuda.stream(stream):
                    b.count_async(opts=o)
                    graph.replay()
                assert b.count_wait() == want_h
                assert a.count_wait() == want
                with torch.cuda.stream(stream):
                    a.count_async(opts=o)
                    graph.replay()
                assert a.count_wait() == want
        finally:
            recorded.clear()
            a.free()
            b.free()
