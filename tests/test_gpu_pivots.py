"""The fused count's pivot structures and work units at their edges, against the oracle."""
import numpy as np
import pytest

import oracle
from bbtc_b200 import Graph, count_batch, graphs, options

pytestmark = pytest.mark.gpu


def wide_rows(n, rows, ids, seed):
    """Rows 0 .. rows-1 (all other rows are empty): each later one of them with
    probability 1/2, and `ids` ids from a shared pool spread over [rows, n), so
    that rows overlap and span the whole id range."""
    rng = np.random.default_rng(seed)
    pool = np.unique(rng.integers(rows, n, size=2 * ids))
    out, indptr = [], np.zeros(n + 1, np.uint32)
    for u in range(rows):
        near = np.arange(u + 1, rows)[rng.random(rows - u - 1) < 0.5]
        row = np.concatenate([near, rng.choice(pool, size=min(ids, len(pool)), replace=False)])
        out.append(np.sort(row))
        indptr[u + 1] = indptr[u] + len(row)
    indptr[rows + 1:] = indptr[rows]
    return graphs.OrientedCSR(n, indptr, np.concatenate(out).astype(np.uint32))


@pytest.mark.parametrize("bitmap_words", [0, 256, 768])
@pytest.mark.parametrize("n,rows,ids", [(1000, 33, 5), (20_000, 40, 20), (1 << 19, 64, 30), (1 << 22, 70, 3),
                                        (1 << 22, 90, 100), (1 << 22, 65, 300)])
def test_wide_pivots(ctx, n, rows, ids, bitmap_words):
    """Bitmap, rank, hash, search and shared-table pivots, and the buffer clean
    between them, for one unit size after the other."""
    g = wide_rows(n, rows, ids, seed=ids)
    for P in (1, 5):
        cuts = graphs.cuts(g, P, "n1d")
        want = oracle.count(g.n, g.indptr, g.indices, cuts)
        assert want > 0
        st = Graph.from_csr(ctx, g, cuts)
        try:
            st.validate()
            for work in (0, 1, 1 << 20):
                o = options(bitmap_words=bitmap_words, unit_work=work, blocks_per_sm=1)
                assert [st.count(opts=o) for _ in range(2)] == [want] * 2, (P, work)
        finally:
            st.free()


@pytest.mark.parametrize("m", [1, 31, 32, 33, 63, 64, 65, 127, 129])
def test_entry_counts_around_a_batch(ctx, m):
    """Dense little graphs cut to m edges: the last batch of every length."""
    edges = [(a, b) for b in range(1, 20) for a in range(b)][:m]
    g = graphs.from_pairs(25, [a for a, _ in edges], [b for _, b in edges])
    cuts = graphs.cuts(g, 3, "uni")
    want = oracle.count(g.n, g.indptr, g.indices, cuts)
    st = Graph.from_csr(ctx, g, cuts)
    two = Graph.from_csr(ctx, g, graphs.cuts(g, 1, "uni"))
    try:
        st.validate()
        assert st.count() == want
        assert count_batch(ctx, [st, two, st]) == [want] * 3
    finally:
        st.free()
        two.free()


@pytest.mark.parametrize("first,second", [({}, {}), ({}, {"kernel": "merge"}), ({"kernel": "search"}, {}),
                                          ({"kernel": "search", "mode": "plain"}, {}),
                                          ({"kernel": "bitmap"}, {"kernel": "merge", "mode": "plain"})])
def test_counts_in_flight_keep_apart(ctx, first, second):
    """Two graphs and an empty one counted before any is waited for: each wait
    returns its graph's last count, whichever was launched last."""
    csrs = [wide_rows(3000, 40, 20, seed=1), wide_rows(3000, 50, 30, seed=2)]
    want = [oracle.count(g.n, g.indptr, g.indices, graphs.cuts(g, 4, "n1d")) for g in csrs] + [0]
    assert want[0] != want[1]
    csrs.append(graphs.OrientedCSR(7, np.zeros(8, np.uint32), np.zeros(0, np.uint32)))
    sts = [Graph.from_csr(ctx, g, graphs.cuts(g, 4, "n1d")) for g in csrs]
    a, b = options(**first), options(**second)
    try:
        for order in ((0, 1, 2), (2, 1, 0), (1, 2, 0)):
            for i in order:
                sts[i].count_async(opts=a)
            for i in (0, 1, 2, 1, 0):
                assert sts[i].count_wait() == want[i], (order, i)
            for i in order:
                sts[i].count_async(opts=b)
                sts[i].count_async(opts=a)
                sts[i].count_async(opts=b)
            assert [st.count_wait() for st in sts] == want, order
            assert count_batch(ctx, sts, a) == want
    finally:
        for st in sts:
            st.free()
