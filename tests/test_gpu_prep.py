"""Device-side preparation equals the host pipeline bit for bit."""
import ctypes

import numpy as np
import pytest

import oracle
from bbtc_b200 import BBTcError, core, graphs

pytestmark = pytest.mark.gpu


class _DeviceView:
    """A zero-copy view of library-owned device memory for torch.as_tensor."""

    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<i4", "data": (ptr, False), "version": 3}


def device_u32(torch, ptr, n):
    return torch.as_tensor(_DeviceView(ptr, n), device="cuda").cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("scale,ef,seed", [(8, 8, 1), (12, 16, 2), (16, 16, 1)])
def test_device_rmat_and_orient_equal_host(ctx, scale, ef, seed):
    torch = pytest.importorskip("torch")
    host = graphs.rmat(scale, ef, seed=seed)
    m_raw = ef << scale
    src = torch.empty(m_raw, dtype=torch.int32, device="cuda")
    dst = torch.empty(m_raw, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    core.rmat_device(ctx, scale, ef, src.data_ptr(), dst.data_ptr(), seed)
    dev = core.DeviceCSR(ctx, 1 << scale, src.data_ptr(), dst.data_ptr(), m_raw)
    assert dev.n == host.n and dev.m == host.m
    torch.cuda.synchronize()
    assert np.array_equal(device_u32(torch, dev.indptr_ptr, dev.n + 1), host.indptr)
    assert np.array_equal(device_u32(torch, dev.indices_ptr, dev.m), host.indices)
    cuts = graphs.cuts(host, 8, "uni")
    g = dev.graph(cuts)
    assert g.count() == oracle.count(host.n, host.indptr, host.indices, cuts)
    g.free()
    dev.free()


def test_orient_device_cleans_pairs(ctx):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(3)
    n = 3000
    src = rng.integers(0, n, size=40000).astype(np.uint32)
    dst = rng.integers(0, n, size=40000).astype(np.uint32)
    src[:100] = dst[:100]  # self-loops
    src = np.concatenate([src, dst[:500], [n + 5]]).astype(np.uint32)  # reversed repeats, an id >= n
    dst = np.concatenate([dst, src[:500], [1]]).astype(np.uint32)
    host = graphs.from_pairs(n, src[:-1], dst[:-1])
    s = torch.from_numpy(src.view(np.int32)).cuda()
    d = torch.from_numpy(dst.view(np.int32)).cuda()
    torch.cuda.synchronize()
    dev = core.DeviceCSR(ctx, n, s.data_ptr(), d.data_ptr(), len(src))
    assert dev.m == host.m
    cuts = graphs.cuts(host, 5, "uni")
    g = dev.graph(cuts)
    assert g.count() == oracle.count(host.n, host.indptr, host.indices, cuts)
    g.free()
    dev.free()


@pytest.mark.parametrize("make", [lambda: graphs.rmat(8, 8, seed=1), lambda: graphs.rmat(16, 16, seed=2),
                                  lambda: graphs.rgg(1 << 14, seed=4),
                                  lambda: graphs.chung_lu(1 << 15, seed=5, max_deg=3000)])
def test_cuts_on_device_equal_host(ctx, make):
    """bbtc_cuts_device (the partitioner on the GPU) gives the host partitioners'
    cuts on the same CSR, for every kind and several stripe counts."""
    torch = pytest.importorskip("torch")
    g = make()
    ip = torch.from_numpy(g.indptr.view(np.int32)).cuda()
    ix = torch.from_numpy(g.indices.view(np.int32)).cuda()
    torch.cuda.synchronize()
    for kind in ("uni", "n1d", "pal"):
        for P in (1, 2, 5, 16, 64):
            got = core.cuts_device(ctx, kind, g.n, ip.data_ptr(), ix.data_ptr(), g.m, P)
            want = graphs.cuts(g, P, kind)
            assert np.array_equal(got, want), (kind, P, got, want)


def test_orient_device_memory(ctx):
    """Preparation holds 36 bytes a pair at most: two arrays of keys (16) and a
    sort's own copy (8) throughout, and beside them the degrees' arrays and then
    the result (4) and the last sort's copy (8).  32 bytes a vertex; 8 MiB of
    histograms and rounding."""
    torch = pytest.importorskip("torch")
    rt = ctypes.CDLL("libcudart.so.12")
    pool = ctypes.c_void_p()
    assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    USED, USED_HIGH = 7, 8  # cudaMemPoolAttrUsedMemCurrent, cudaMemPoolAttrUsedMemHigh

    def attr(which):
        v = ctypes.c_uint64()
        assert rt.cudaMemPoolGetAttribute(pool, which, ctypes.byref(v)) == 0
        return v.value

    n, m = 1 << 16, 1 << 22
    s, d = (torch.randint(0, n, (m,), dtype=torch.int32, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    before = attr(USED)
    assert rt.cudaMemPoolSetAttribute(pool, USED_HIGH, ctypes.byref(ctypes.c_uint64(0))) == 0
    dev = core.DeviceCSR(ctx, n, s.data_ptr(), d.data_ptr(), m)
    peak = attr(USED_HIGH) - before
    print(f"{peak / m:.2f} bytes a pair")
    assert dev.m > m * 9 // 10
    dev.free()
    assert peak <= 36 * m + 32 * n + (8 << 20)


def test_failed_preparation_holds_nothing(ctx):
    """Each device allocation of a preparation fails in turn: BBTC_ERR_NOMEM, and
    the device's pool holds what it held before."""
    torch = pytest.importorskip("torch")
    rt = ctypes.CDLL("libcudart.so.12")
    pool = ctypes.c_void_p()
    assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0

    def used():
        torch.cuda.synchronize()
        v = ctypes.c_uint64()
        assert rt.cudaMemPoolGetAttribute(pool, 7, ctypes.byref(v)) == 0  # cudaMemPoolAttrUsedMemCurrent
        return v.value

    n, m = 1000, 20000
    s, d = (torch.randint(0, n, (m,), dtype=torch.int32, device="cuda") for _ in range(2))
    before = used()
    try:
        for k in range(100):
            core.debug_fail_alloc(k)
            try:
                dev = core.DeviceCSR(ctx, n, s.data_ptr(), d.data_ptr(), m)
            except BBTcError as e:
                assert e.status == -3, (k, e.message)
                assert used() == before, k
                continue
            assert core.debug_fail_alloc(-1) >= 0  # every allocation passed
            dev.free()
            break
        assert 5 < k < 99
        assert used() == before
    finally:
        core.debug_fail_alloc(-1)
