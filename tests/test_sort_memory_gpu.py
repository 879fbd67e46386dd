"""A pair sort where device memory holds one pair of temporaries but not two: the calling program's memory
pool is limited to 192 MiB, of which 16,777,216 pairs (three passes) take 256 MiB with two pairs of
temporaries and 128 MiB with one, besides 13 MiB of sort scratch."""
from __future__ import annotations

import ctypes as C

import pytest

from vkfluidsim_gb300 import primitives

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


class _PoolProps(C.Structure):  # CUmemPoolProps
    _fields_ = [("alloc_type", C.c_int), ("handle_types", C.c_int), ("location_type", C.c_int),
                ("location_id", C.c_int), ("win32", C.c_void_p), ("max_size", C.c_size_t),
                ("usage", C.c_ushort), ("reserved", C.c_ubyte * 54)]


@pytest.fixture
def limited_pool():
    torch.zeros(1, device="cuda")
    cu = C.CDLL("libcuda.so.1")
    dev = C.c_int(torch.cuda.current_device())

    def ok(code):
        assert code == 0, code

    before, pool = C.c_void_p(), C.c_void_p()
    ok(cu.cuDeviceGetMemPool(C.byref(before), dev))
    props = _PoolProps(alloc_type=1, location_type=1, location_id=dev.value, max_size=192 << 20)
    ok(cu.cuMemPoolCreate(C.byref(pool), C.byref(props)))
    ok(cu.cuDeviceSetMemPool(dev, pool))
    yield
    torch.cuda.synchronize()
    ok(cu.cuDeviceSetMemPool(dev, before))
    ok(cu.cuMemPoolDestroy(pool))


@pytest.mark.parametrize("max_value", [(1 << 24) - 1, (1 << 32) - 1])  # three passes, four passes
def test_sort_with_one_pair_of_temporaries(limited_pool, max_value):
    n = 1 << 24
    keys = torch.randint(0, min(max_value, 2**31 - 1), (n,), dtype=torch.int32, device="cuda")
    want, perm = torch.sort(keys, stable=True)
    items = torch.empty_like(keys)
    s = torch.cuda.current_stream().cuda_stream
    primitives.sort_pairs(items.data_ptr(), keys.data_ptr(), n, max_value, s)
    torch.cuda.synchronize()
    assert torch.equal(keys, want) and torch.equal(items, perm.to(torch.int32))
    assert primitives.sort_status() == 0
