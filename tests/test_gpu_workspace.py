"""Device memory that a call takes beside the graph (the high-water mark of the
device's stream-ordered pool): bounds from the arrays that each call needs."""
import ctypes

import pytest

import hornet_b200 as H

pytestmark = pytest.mark.gpu

USED_CURRENT, USED_HIGH = 7, 8   # CU_MEMPOOL_ATTR_USED_MEM_*


def peak(call):
    """Bytes of the pool in use at the call's peak beyond those before it."""
    import torch
    torch.cuda.synchronize()
    cu = ctypes.CDLL("libcuda.so.1")
    pool, v = ctypes.c_void_p(), ctypes.c_uint64(0)
    assert cu.cuDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    assert cu.cuMemPoolSetAttribute(pool, USED_HIGH, ctypes.byref(v)) == 0
    assert cu.cuMemPoolGetAttribute(pool, USED_CURRENT, ctypes.byref(v)) == 0
    before = v.value
    call()
    torch.cuda.synchronize()
    assert cu.cuMemPoolGetAttribute(pool, USED_HIGH, ctypes.byref(v)) == 0
    return v.value - before


def rmat(scale, ef):
    import torch
    n = ef << scale
    s = torch.empty(n, dtype=torch.int32, device="cuda")
    d = torch.empty_like(s)
    H.gen_rmat_device(scale, n, 5, s, d)
    torch.cuda.synchronize()
    return H.hornet_from_device_csr(H.coo_to_csr_device(1 << scale, s, d))


@pytest.mark.parametrize("scale", [16, 18])   # by id, by rank
@pytest.mark.parametrize("flip,cap", [(1, 16384), (1, 64), (0, 16384)])
def test_triangle_counts(scale, flip, cap):
    h = rmat(scale, 40)
    m, n = h.nE(), h.nV()
    tc = H.TriangleCounting2(h)
    # lists, candidates and their slots hold the oriented half of the edges (and
    # up to three pads a vertex); 1 byte an edge of work items, direction bits
    # and tile counters; offsets, degrees, counters and the rank sort a vertex.
    # Without bitmaps a flag an edge is scanned before.
    bound = 7 * m + 110 * n + (16 << 20)
    try:
        H.tune_set("tc.flip", flip)
        H.tune_set("tc.cta_table_cap", cap)
        assert peak(tc.run) < bound
    finally:
        H.tune_reset()


@pytest.mark.parametrize("n", [(1 << 20) + 1, 3_000_003])
def test_large_updates(n):
    """Keys twice, their places and counters (32 bytes an entry) and the plan's
    arrays (48); the list of hubs takes the keys' place."""
    import torch
    h = rmat(18, 16)
    s = torch.empty(n, dtype=torch.int32, device="cuda")
    d = torch.empty_like(s)
    H.gen_rmat_device(18, n, 9, s, d, a=0.25, b=0.25, c=0.25)
    torch.cuda.synchronize()
    b = H.BatchUpdate(h, s, d)
    assert peak(lambda: h.insert(b, True, True)) < 81 * n
    assert peak(lambda: h.erase(b, True)) < 81 * n


def test_updates_without_room_for_one_allocation():
    """2^20 entries with 120 MB free: too little for the one allocation of all
    buffers (151 MB), enough for the buffers one by one (84 MB)."""
    import numpy as np
    import torch
    h = rmat(18, 8)
    n = 1 << 20
    # edges that the graph does not hold: from isolated vertices
    src, dst = h.getCOO(True)
    isolated = np.flatnonzero(np.bincount(src, minlength=h.nV()) == 0).astype(np.int32)
    rng = np.random.default_rng(3)
    s = torch.from_numpy(isolated[rng.integers(0, len(isolated), n)]).cuda()
    d = torch.from_numpy(rng.integers(0, h.nV(), n).astype(np.int32)).cuda()
    torch.cuda.synchronize()
    b = H.BatchUpdate(h, s, d)
    cu = ctypes.CDLL("libcuda.so.1")
    pool = ctypes.c_void_p()
    assert cu.cuDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    assert cu.cuMemPoolTrimTo(pool, ctypes.c_size_t(0)) == 0
    torch.cuda.empty_cache()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - (120 << 20), dtype=torch.uint8, device="cuda")
    try:
        assert torch.cuda.mem_get_info()[0] < 150 << 20
        assert h.erase(b) == 0
        assert h.nE() == len(src)
    finally:
        del hog
        torch.cuda.empty_cache()
    assert h.erase(b) == 0
