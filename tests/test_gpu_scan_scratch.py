"""The carry scans' scratch: what one scan leaves there never matters to the next."""
import numpy as np
import pytest

from gpu_util import to_dev, to_host
from natural_number_gb300.synth import limbs

pytestmark = pytest.mark.gpu


def empty(n):
    import torch
    return torch.empty(n, dtype=torch.uint64, device="cuda")


@pytest.mark.parametrize("na,nb", [(1000, 25), (1985, 64), (1986, 64), (65500, 31), (65530, 31), (131072, 16),
                                   ((1 << 20) + 3, 3), (3 << 20, 2)])
def test_long_base_case(oracle, na, nb):
    """Tiles of both lengths, a last tile of one position; carries that cross
    every tile: (B^na - 1) * 1 + runs, and all ones."""
    import natural_number_gb300 as nn
    ctx = nn.Context(0)
    ones = np.full(na, 2**64 - 1, dtype=np.uint64)
    b = limbs(nb, nb)
    one = np.zeros(nb, dtype=np.uint64)
    one[0] = 1
    out = empty(na + nb)
    for x, y in ((limbs(na, na), b), (ones, np.full(nb, 2**64 - 1, dtype=np.uint64)), (ones, b), (ones, one)):
        ctx.mul_base_device(out, to_dev(x), to_dev(y))
        ctx.synchronize()
        got, want = to_host(out), oracle.mul_base(x, y)
        assert np.array_equal(got[: want.size], want) and not got[want.size:].any()
    ctx.close()


def test_products_after_overlapping_ones(oracle):
    """Two products of one context on two streams at once may spoil each other,
    but nothing that comes after them."""
    import torch
    import natural_number_gb300 as nn
    na, nb = 30000, 25
    a, b = limbs(1, na), limbs(2, nb)
    da, db, want = to_dev(a), to_dev(b), oracle.mul(a, b)
    ctx = nn.Context(0)
    outs = [empty(na + nb) for _ in range(3)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for _ in range(50):
        for s, o in zip(streams, outs):
            ctx.set_stream(s.cuda_stream)
            ctx.mul_base_device(o, da, db)
    torch.cuda.synchronize()
    for _ in range(3):
        ctx.mul_base_device(outs[2], da, db)
        ctx.synchronize()
        assert np.array_equal(to_host(outs[2])[: want.size], want)
    ctx.set_stream(None)
    ctx.close()
