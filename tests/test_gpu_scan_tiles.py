"""Carry scans at the edges of their tile rules (one cluster, tiles of 512, tiles
of 2048): sums and products whose carries run through whole tiles."""
import numpy as np
import pytest

from gpu_util import to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2047, 2048, 2049, 8191, 8193, 65535, 65536, 65537, 70001])
def test_carries_through_tiles(oracle, n):
    import torch
    import natural_number_gb300 as nn
    ctx = nn.Context(0)
    ones = np.full(n, 2**64 - 1, dtype=np.uint64)
    short = np.full(n // 3 + 1, 2**64 - 1, dtype=np.uint64)
    low = np.zeros(n, dtype=np.uint64)
    low[0], low[n - 1] = 1, 1
    for a, b in [(ones, ones), (ones, short), (low, ones), (ones, low)]:
        out = torch.empty(a.size + b.size, dtype=torch.uint64, device="cuda")
        ctx.mul_device(out, to_dev(a), to_dev(b))
        ctx.synchronize()
        got, want = to_host(out), oracle.mul(a, b)
        assert np.array_equal(got[: want.size], want) and not got[want.size:].any()
    # (B^n - 1) x + r with x near a power: a quotient of runs of ones
    num = np.concatenate([ones, short])
    q = torch.empty(num.size - n + 1, dtype=torch.uint64, device="cuda")
    r = torch.empty(n, dtype=torch.uint64, device="cuda")
    div = ones.copy()
    div[0] = 12345
    ctx.div_device(q, r, to_dev(num), to_dev(div))
    ctx.synchronize()
    value = lambda x: int.from_bytes(np.ascontiguousarray(x).tobytes(), "little")
    hq, hr = to_host(q), to_host(r)
    assert value(oracle.mul(hq, div)) + value(hr) == value(num) and value(hr) < value(div)
    ctx.close()
