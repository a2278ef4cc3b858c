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
