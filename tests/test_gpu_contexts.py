"""One context's options do not reach another context's launches."""
import pytest

import oracle
from bbtc_b200 import Context, Graph, graphs, options

pytestmark = pytest.mark.gpu


def workload(seed):
    g = graphs.rmat(10, 16, seed=seed)
    cuts = graphs.cuts(g, 4, "uni")
    return g, cuts, oracle.count(g.n, g.indptr, g.indices, cuts)


@pytest.mark.parametrize("kernel,mode", [("fused", "persistent"), ("bitmap", "persistent"), ("search", "plain")])
def test_buffer_sizes_of_two_contexts(kernel, mode):
    """A context that counts with a large shared buffer still does after a new
    context has counted with a small one."""
    g, cuts, want = workload(21)
    large = options(kernel=kernel, mode=mode, bitmap_words=4096)
    small = options(kernel=kernel, mode=mode, bitmap_words=256)
    with Context(0) as a, Context(0) as b:
        st = [Graph.from_csr(c, g, cuts) for c in (a, b)]
        try:
            for _ in range(2):
                assert st[0].count(opts=large) == want
                assert st[1].count(opts=small) == want
        finally:
            for x in st:
                x.free()
