"""The block CSRs of the per-task kernels at the edges of their builder's batches, on random CSRs."""
import numpy as np
import pytest

import oracle
from bbtc_b200 import Graph, graphs, options

pytestmark = pytest.mark.gpu


def csr(n, degrees, m, oriented, seed):
    """m edges: rows in a shuffled order get degrees[i % len(degrees)] ids each
    until there are m edges; ids above the row, or anywhere."""
    rng = np.random.default_rng(seed)
    rows = [np.zeros(0, np.int64)] * n
    left = m
    for i, u in enumerate(rng.permutation(n)):
        room = n - 1 - u if oriented else n
        d = min(degrees[i % len(degrees)], int(room), left)
        rows[u] = np.sort(rng.choice(int(room), size=d, replace=False)) + (u + 1 if oriented else 0)
        left -= d
    assert left == 0
    indptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.uint32)
    return graphs.OrientedCSR(n, indptr, np.concatenate(rows).astype(np.uint32))


CASES = [  # vertices, degrees, edges
    (3, [2], 3), (40, [31], 127), (40, [31], 128), (40, [31], 129), (300, [1, 0, 0, 5], 255),
    (300, [200], 257),             # runs longer than a warp's edges
    (5000, [0] * 60 + [90], 4096), # more than 32 empty rows in a row
    (3000, [2500, 3, 0], 40_001),  # runs of thousands of edges
]


@pytest.mark.parametrize("oriented", [True, False])
@pytest.mark.parametrize("n,degrees,m", CASES)
def test_block_csrs(ctx, n, degrees, m, oriented):
    g = csr(n, degrees, m, oriented, seed=m)
    for cuts in ([0, n], [0, 0, n // 3, n // 3, n + 9], list(range(0, 63)) + [max(62, n // 2), max(62, n)]):
        cuts = np.array(cuts, np.uint32)
        want = oracle.count(g.n, g.indptr, g.indices, cuts)
        for first, second in (("bitmap", "merge"), ("merge", "search")):  # both at once, or the forward one first
            st = Graph.from_csr(ctx, g, cuts)
            try:
                assert st.count(opts=options(kernel=first)) == want
                st.validate()
                assert st.count(opts=options(kernel=second)) == want
                st.validate()
            finally:
                st.free()
