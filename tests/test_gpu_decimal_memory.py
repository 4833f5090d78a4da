"""A decimal conversion in a memory pool that holds a level of its split but not
what the faster way holds beyond it: the powers of all levels and the level
before's plans."""
import ctypes

import pytest

from natural_number_gb300.synth import limbs

pytestmark = pytest.mark.gpu


class PoolProps(ctypes.Structure):  # CUmemPoolProps
    _fields_ = [("alloc_type", ctypes.c_int), ("handle_types", ctypes.c_int), ("location_type", ctypes.c_int),
                ("location_id", ctypes.c_int), ("security", ctypes.c_void_p), ("max_size", ctypes.c_size_t),
                ("usage", ctypes.c_ushort), ("reserved", ctypes.c_ubyte * 54)]


def test_conversion_in_a_small_pool():
    import torch
    import natural_number_gb300 as nn
    a = limbs(7, 1000003)
    ctx = nn.Context(0)
    want = ctx.to_dec_levels(a)  # powers and tables are there
    cu = ctypes.CDLL("libcuda.so.1")
    default, pool = ctypes.c_void_p(), ctypes.c_void_p()
    assert cu.cuDeviceGetMemPool(ctypes.byref(default), 0) == 0
    # pinned memory of device 0, at most 190 MB: a level's products alone take 162, with all that is held 225
    props = PoolProps(alloc_type=1, location_type=1, location_id=0, max_size=190 << 20)
    assert cu.cuMemPoolCreate(ctypes.byref(pool), ctypes.byref(props)) == 0
    assert cu.cuDeviceSetMemPool(0, pool) == 0
    try:
        assert ctx.to_dec_levels(a) == want
    finally:
        torch.cuda.synchronize()
        assert cu.cuDeviceSetMemPool(0, default) == 0
        cu.cuMemPoolDestroy(pool)
    assert ctx.to_dec_levels(a) == want
    ctx.close()
