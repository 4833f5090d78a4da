"""The carry scans' scratch: what a scan finds there never matters to the next
one, and a captured graph keeps the words it was captured with when a longer
scan of the same context wants more."""
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


@pytest.mark.parametrize("na,nb", [(20000, 20), (3000, 2500), (400000, 300000)])
def test_replay_after_the_scratch_grew(oracle, na, nb):
    import torch
    import natural_number_gb300 as nn
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        ctx = nn.Context(0)
        x, y, out = empty(na), empty(nb), empty(na + nb)
        x.copy_(to_dev(limbs(1, na)))
        y.copy_(to_dev(limbs(2, nb)))
        ctx.mul_device(out, x, y)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            ctx.mul_device(out, x, y)
        long = torch.randint(-(2**63), 2**63 - 1, (1 << 22,), dtype=torch.int64, device="cuda").view(torch.uint64)
        t = empty(1 << 23)
        ctx.mul_device(t, long, long)  # 4096 tiles: more than the scratch held
        for seed in (3, 5):
            a, b = limbs(seed, na), limbs(seed + 1, nb)
            x.copy_(to_dev(a))
            y.copy_(to_dev(b))
            graph.replay()
            stream.synchronize()
            want = oracle.mul(a, b)
            assert np.array_equal(to_host(out)[: want.size], want)
        ctx.close()
