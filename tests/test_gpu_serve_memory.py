"""Device memory of the request server: batches of short products, with one of a
longer transform among them, stay within the budget that admits them."""
import ctypes

import numpy as np
import pytest

from natural_number_gb300.synth import limbs

pytestmark = pytest.mark.gpu

USED_CURRENT, USED_HIGH = 7, 8  # CUmemPool_attribute


def _pool():
    cu = ctypes.CDLL("libcuda.so.1")
    pool = ctypes.c_void_p()
    assert cu.cuDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0

    def read(attribute):
        v = ctypes.c_uint64()
        assert cu.cuMemPoolGetAttribute(pool, attribute, ctypes.byref(v)) == 0
        return v.value

    def reset():
        assert cu.cuMemPoolSetAttribute(pool, USED_HIGH, ctypes.byref(ctypes.c_uint64(0))) == 0

    return read, reset


@pytest.mark.parametrize("small", [(64, 200), (200, 250)])
def test_short_products_stay_within_the_budget(oracle, small):
    import natural_number_gb300 as nn
    budget = 1 << 20
    srv = nn.Server(0, hbm_budget=budget, streams=1, div_workers=1)
    long = (limbs(1, 2000), limbs(2, 2000))
    srv.wait(srv.submit_mul(*long))  # the tables are there
    read, reset = _pool()
    base = read(USED_CURRENT)
    reset()
    jobs = [long if k % 25 == 0 else (limbs(2 * k, small[0]), limbs(2 * k + 1, small[1])) for k in range(400)]
    tickets = [srv.submit_mul(a, b) for a, b in jobs]
    results = [srv.wait(t) for t in tickets]
    high = read(USED_HIGH)
    stats = srv.stats()
    srv.close()
    for (a, b), (got, _) in zip(jobs, results):
        assert np.array_equal(got, oracle.mul(a, b))
    assert stats["peak_bytes"] <= budget
    # freed memory counts until its stream gets there: one batch more at most
    assert high - base <= 2 * budget
