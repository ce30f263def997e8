"""Coulomb and exchange past N = 512, where a row of K is longer than a block's positions.  No
memory holds such a tensor, so its N slabs are one: T[p,q,r,s] = t[q,r,s], a slab of 1000 pages of
2 MiB for N = 640, mapped N times in a row."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

N = 640
PAGE = 2 << 20


class _Location(ctypes.Structure):
    _fields_ = [("type", ctypes.c_int), ("id", ctypes.c_int)]


class _AllocProp(ctypes.Structure):  # CUmemAllocationProp
    _fields_ = [("type", ctypes.c_int), ("handles", ctypes.c_int), ("location", _Location), ("win32", ctypes.c_void_p),
                ("compression", ctypes.c_ubyte), ("rdma", ctypes.c_ubyte), ("usage", ctypes.c_ushort),
                ("reserved", ctypes.c_ubyte * 4)]


class _AccessDesc(ctypes.Structure):
    _fields_ = [("location", _Location), ("flags", ctypes.c_int)]


def _fill(ptr, g):
    """The slab's values, copied in from a torch tensor."""
    import torch
    t = torch.randn(N ** 3, generator=g, device="cuda", dtype=torch.float64)
    drv = ctypes.CDLL("libcuda.so.1")
    assert drv.cuMemcpyDtoD_v2(ctypes.c_uint64(ptr), ctypes.c_uint64(t.data_ptr()), ctypes.c_size_t(8 * N ** 3)) == 0
    return t.view(N, N, N)


def test_rows_longer_than_a_block():
    import torch
    from mmd import _native
    torch.cuda.init()
    torch.zeros(1, device="cuda")
    drv = ctypes.CDLL("libcuda.so.1")
    slab = 8 * N ** 3
    assert slab % PAGE == 0
    loc = _Location(1, torch.cuda.current_device())  # CU_MEM_LOCATION_TYPE_DEVICE
    prop = _AllocProp(type=1, location=loc)          # CU_MEM_ALLOCATION_TYPE_PINNED
    gran, handle, base = ctypes.c_size_t(), ctypes.c_uint64(), ctypes.c_uint64()
    assert drv.cuMemGetAllocationGranularity(ctypes.byref(gran), ctypes.byref(prop), 0) == 0
    if PAGE % gran.value:
        pytest.skip("allocation granularity above 2 MiB")
    assert drv.cuMemCreate(ctypes.byref(handle), ctypes.c_size_t(slab), ctypes.byref(prop), ctypes.c_ulonglong(0)) == 0
    mapped = 0
    try:
        assert drv.cuMemAddressReserve(ctypes.byref(base), ctypes.c_size_t(slab * N), ctypes.c_size_t(0),
                                       ctypes.c_uint64(0), ctypes.c_ulonglong(0)) == 0
        for k in range(N):
            assert drv.cuMemMap(ctypes.c_uint64(base.value + k * slab), ctypes.c_size_t(slab), ctypes.c_size_t(0), handle,
                                ctypes.c_ulonglong(0)) == 0
            mapped += 1
        access = _AccessDesc(loc, 3)                 # CU_MEM_ACCESS_FLAGS_PROT_READWRITE
        assert drv.cuMemSetAccess(base, ctypes.c_size_t(slab * N), ctypes.byref(access), ctypes.c_size_t(1)) == 0
        g = torch.Generator(device="cuda").manual_seed(N)
        t = _fill(base.value, g)
        P = torch.randn(N, N, generator=g, device="cuda", dtype=torch.float64)
        J, K = torch.empty_like(P), torch.empty_like(P)
        p = lambda x: ctypes.c_void_p(x.data_ptr())
        _native.check(_native.lib().mmdg_jk_dense(_native.scratch_context()._h, N, ctypes.c_void_p(base.value), p(P), p(J),
                                                  p(K), _native.stream_ptr()), "mmdg_jk_dense")
        torch.cuda.synchronize()
        Jr = (t.reshape(N, -1) @ P.T.reshape(-1)).expand(N, N)     # J_pq = sum_rs t_qrs P_sr
        Kr = torch.einsum("sqr,sr->q", t, P).expand(N, N)          # K_pq = sum_rs t_sqr P_sr
        # N^2 products of unit normals, each summed with a relative rounding of 1.1e-16, both sides
        tol = 2.4e-16 * N * N * 12.0
        assert float((J - Jr).abs().max()) < tol and float((K - Kr).abs().max()) < tol
    finally:
        torch.cuda.synchronize()
        for k in range(mapped):
            drv.cuMemUnmap(ctypes.c_uint64(base.value + k * slab), ctypes.c_size_t(slab))
        if base.value:
            drv.cuMemAddressFree(base, ctypes.c_size_t(slab * N))
        drv.cuMemRelease(handle)
