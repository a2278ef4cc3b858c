"""A server of per-task counts holds budget for the block CSRs that they read."""
import pytest

import oracle
from bbtc_b200 import Context, Graph, Server, core, graphs, options

pytestmark = pytest.mark.gpu


def load_bytes(n, m, cuts):
    """Upper bound of a per-task request while it is loaded (the server's estimate)."""
    P = len(cuts) - 1
    rp = sum(P * ((int(b) - int(a) + 1 + 3) & ~3) for a, b in zip(cuts[:-1], cuts[1:]))
    lists = 16 * m + m // 8 + 32 * (min(n, m) + 1)
    temps = 32 * m + 16 * (n + 4) + (16 << 20)
    return (4 * (n + 1) + 4 * m + lists + temps + 12 * (rp + 4) + 8 * (m + 4 * P * P + 4)
            + 8 * (m // 32 + 2 * P * P + 2))


@pytest.mark.parametrize("kernel", ["bitmap", "merge"])
def test_ready_graphs_hold_their_tiles(kernel):
    g = graphs.rmat(17, 16, seed=31)
    cuts = graphs.cuts(g, 48, "uni")
    want = oracle.count(g.n, g.indptr, g.indices, cuts)
    o = options(kernel=kernel)
    with Context(0) as ctx:
        st = Graph.from_csr(ctx, g, cuts)
        bare = st.info().device_bytes
        assert st.count(opts=o) == want
        held = st.info().device_bytes
        st.free()
    tiles = held - bare
    assert tiles > 4 * g.m
    one = load_bytes(g.n, g.m, cuts)
    # one request held and one loading fit without the held one's tiles, and do not with them
    with Server(0, hbm_budget=bare + one + tiles // 2, loaders=2, opts=o) as srv:
        ids = [srv.submit_csr(g, cuts) for _ in range(4)]
        infos = [srv.wait(r, 60000) for r in ids]
        for r in ids:
            srv.release(r)
    assert [(i.status, i.count) for i in infos] == [(1, want)] * 4
    infos.sort(key=lambda i: i.load_ns)
    for a, b in zip(infos[:-1], infos[1:]):
        assert b.load_ns >= a.done_ns  # the next load starts when the last request has given its memory back


def test_per_task_request_fails_alone():
    """An allocation that fails while the block CSRs are built fails that
    request and holds nothing."""
    g = graphs.rmat(10, 16, seed=11)
    cuts = graphs.cuts(g, 4, "uni")
    want = oracle.count(g.n, g.indptr, g.indices, cuts)
    with Server(0, loaders=1, opts=options(kernel="bitmap")) as srv:
        for k in range(100):
            core.debug_fail_alloc(k)
            rid = srv.submit_csr(g, cuts)
            info = srv.wait(rid, 60000)
            srv.release(rid)
            if core.debug_fail_alloc(-1) >= 0:
                assert (info.status, info.count) == (1, want)
                break
            assert info.status == -3, (k, info.status)
            ok = srv.submit_csr(g, cuts)
            info = srv.wait(ok, 60000)
            srv.release(ok)
            assert (info.status, info.count) == (1, want), k
            assert srv.stats().device_bytes_in_use == 0, k
        else:
            pytest.fail("a request made more than 100 device allocations")
        assert k > 8  # more than an upload's own: the block CSRs' too
