"""The layout's single-pass kernels: tiles, waits between them and their ends."""
import numpy as np
import pytest

import oracle
from bbtc_b200 import BBTcError, Graph, graphs

pytestmark = pytest.mark.gpu

TIMEOUT = -5


def bands(n, m):
    """Rows of consecutive ids, of 0 to 60 of them in turn, m edges in all."""
    want = np.minimum(np.arange(n, dtype=np.int64) * 7 % 61, n - 1 - np.arange(n))
    ends = np.minimum(np.cumsum(want), m)
    assert ends[-1] == m
    indptr = np.concatenate([[0], ends]).astype(np.uint32)
    deg = np.diff(indptr.astype(np.int64))
    rows = np.repeat(np.arange(n), deg)
    indices = rows + 1 + np.arange(m) - np.repeat(indptr[:-1].astype(np.int64), deg)
    return graphs.OrientedCSR(n, indptr, indices.astype(np.uint32))


@pytest.mark.parametrize("m", [1 << 13, 1 << 20, (1 << 22) + 1])  # small tiles, large pair tiles, large pivot tiles
@pytest.mark.parametrize("which", [1, 2])
def test_wait_for_a_tile_runs_out(ctx, which, m):
    """The first tile of a pass publishes nothing: the blocks that wait for it
    leave, the upload returns BBTC_ERR_TIMEOUT, and the next one is right."""
    g = bands(m // 25, m)
    cuts = np.array([0, g.n // 3, g.n], np.uint32)
    ctx.debug_layout_timeout(which, 2000)
    try:
        for _ in range(2):
            with pytest.raises(BBTcError) as e:
                Graph.from_csr(ctx, g, cuts)
            assert e.value.status == TIMEOUT, e.value.message
    finally:
        ctx.debug_layout_timeout(0, 0)
    st = Graph.from_csr(ctx, g, cuts)
    try:
        st.validate()
        assert st.count() == oracle.count(g.n, g.indptr, g.indices, cuts)
    finally:
        st.free()


def check(ctx, g, cuts):
    st = Graph.from_csr(ctx, g, cuts)
    try:
        st.validate()
        assert st.count() == oracle.count(g.n, g.indptr, g.indices, np.asarray(cuts, np.uint32))
    finally:
        st.free()


SIZES = [base + d for base in (1 << 20, 1 << 22) for d in (-1, 0, 1)]  # around the edges from which tiles are large


@pytest.mark.parametrize("m", SIZES)
def test_layout_around_the_tile_forms(ctx, m):
    """Pairs and pivots of every tile, the last one full, one edge long or one short."""
    g = bands(m // 25, m)
    check(ctx, g, np.array([0, g.n // 3, g.n // 2, g.n], np.uint32))


@pytest.mark.parametrize("m", SIZES[1::3])
def test_layout_of_large_unoriented(ctx, m):
    """Ids below their rows, above and equal: the passes that go over the lists of all tiles."""
    g = bands(m // 25, m)
    deg = np.diff(g.indptr.astype(np.int64))
    down = np.minimum(deg // 2 + 1, np.arange(g.n))  # every row moved down by half its length or more
    g = graphs.OrientedCSR(g.n, g.indptr, (g.indices - np.repeat(down, deg)).astype(np.uint32))
    check(ctx, g, np.array([0, 7, g.n // 2, g.n + 3], np.uint32))


@pytest.mark.parametrize("n,ids,m", [(150_000, 70_000, 500_000), (600_000, 300_000, 1_500_000)])
def test_rows_across_many_tiles(ctx, n, ids, m):
    """Rows of more than 32 tiles, small and large, so that the nearest row start is past a whole look-back window."""
    rng = np.random.default_rng(ids)
    hubs = [np.sort(rng.choice(n - 3, size=ids, replace=False)) + 3 for _ in range(3)]
    rest = bands(n - 3, m - 3 * ids)
    indptr = np.concatenate([np.arange(3) * ids, rest.indptr.astype(np.int64) + 3 * ids])
    g = graphs.OrientedCSR(n, indptr.astype(np.uint32), np.concatenate(hubs + [rest.indices.astype(np.int64) + 3]).astype(np.uint32))
    check(ctx, g, np.array([0, 2, n // 2, n], np.uint32))


@pytest.mark.parametrize("at", [0, 1 << 19, (1 << 20) + 3])  # in the first, a middle and the last tile
@pytest.mark.parametrize("fault", ["range", "order"])
def test_broken_ids_are_found_in_any_tile(ctx, at, fault):
    m = (1 << 20) + 5
    g = bands(m // 25, m)
    indices = g.indices.copy()
    if fault == "range":
        indices[at] = g.n
    else:  # an id as large as the next one of its row
        while at + 1 in g.indptr:
            at += 1
        indices[at] = indices[at + 1]
    with pytest.raises(BBTcError) as e:
        Graph.upload(ctx, g.n, g.indptr, indices, np.array([0, g.n], np.uint32))
    assert e.value.status == -4, e.value.message
