"""Products and squares of the two longest transforms (2^30 and 2^31 points:
blocks of 256 and 512 coefficients, 2^28 and 2^29 limbs an operand): all ones,
where every sum is as large as it can be, limb by limb, and random limbs modulo
2^64 - 1 and 2^64 + 1.  Checked on the device: the host would copy gigabytes."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

CHUNK = 1 << 26


def value_mod(x):
    """The value of device limbs (int64 words) modulo 2^64 - 1 and 2^64 + 1."""
    every, alternating = 0, 0
    for k in range(0, x.numel(), CHUNK):  # CHUNK is even
        w = x[k:k + CHUNK]
        lo, hi = w & 0xFFFFFFFF, (w >> 32) & 0xFFFFFFFF  # sums of 2^26 stay below 2^58
        even = int(lo[0::2].sum()) + (int(hi[0::2].sum()) << 32)
        odd = int(lo[1::2].sum()) + (int(hi[1::2].sum()) << 32)
        every += even + odd
        alternating += even - odd
    return every % (2**64 - 1), alternating % (2**64 + 1)


def all_ones_product(out, n, m):
    """(B^n - 1)(B^m - 1) = B^(n+m) - B^n - B^m + 1, n >= m."""
    def same(lo, hi, word):
        return all(bool((out[k:min(k + CHUNK, hi)] == word).all()) for k in range(lo, hi, CHUNK))
    if n == m:
        return same(0, 1, 1) and same(1, n, 0) and same(n, n + 1, -2) and same(n + 1, 2 * n, -1)
    return same(0, 1, 1) and same(1, m, 0) and same(m, n, -1) and same(n, n + 1, -2) and same(n + 1, n + m, -1)


@pytest.mark.parametrize("s", [30, 31])
def test_longest(s):
    import torch
    import natural_number_gb300 as nn
    n, m = (1 << (s - 2)) + 3, (1 << (s - 2)) + 1
    g = torch.Generator(device="cuda")
    g.manual_seed(s)
    ctx = nn.Context(0)
    out = torch.empty(2 * n, dtype=torch.int64, device="cuda")
    try:
        a = torch.full((n,), -1, dtype=torch.int64, device="cuda")
        ctx.mul_device(out[: n + m].view(torch.uint64), a.view(torch.uint64), a[:m].view(torch.uint64))
        ctx.synchronize()
        assert all_ones_product(out, n, m)
        ctx.sqr_device(out.view(torch.uint64), a.view(torch.uint64))
        ctx.synchronize()
        assert all_ones_product(out, n, n)
        b = torch.randint(-(2**63), 2**63 - 1, (m,), dtype=torch.int64, device="cuda", generator=g)
        for k in range(0, n, CHUNK):
            e = min(k + CHUNK, n)
            a[k:e] = torch.randint(-(2**63), 2**63 - 1, (e - k,), dtype=torch.int64, device="cuda", generator=g)
        ctx.mul_device(out[: n + m].view(torch.uint64), a.view(torch.uint64), b.view(torch.uint64))
        ctx.synchronize()
        va, vb, vp = value_mod(a), value_mod(b), value_mod(out[: n + m])
        assert vp[0] == va[0] * vb[0] % (2**64 - 1)
        assert vp[1] == va[1] * vb[1] % (2**64 + 1)
        ctx.sqr_device(out.view(torch.uint64), a.view(torch.uint64))
        ctx.synchronize()
        vs = value_mod(out)
        assert vs[0] == va[0] * va[0] % (2**64 - 1)
        assert vs[1] == va[1] * va[1] % (2**64 + 1)
    finally:
        ctx.close()
        del out
        torch.cuda.empty_cache()
        cu, pool = ctypes.CDLL("libcuda.so.1"), ctypes.c_void_p()
        if cu.cuDeviceGetMemPool(ctypes.byref(pool), 0) == 0:  # a hundred gigabytes go back
            cu.cuMemPoolTrimTo(pool, ctypes.c_size_t(0))
