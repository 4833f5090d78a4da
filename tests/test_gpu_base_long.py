"""Base-case products on both sides of every line of their tiles' rule, the
lengths of a tile and of a wave of them: all ones, limbs with long carries, and
the same under capture, where no words are to be had for more tiles."""
import numpy as np
import pytest

from gpu_util import to_dev, to_host
from natural_number_gb300.synth import limbs

pytestmark = pytest.mark.gpu

SHORT, LONG = 56 << 10, 3 << 16


@pytest.mark.parametrize("total,nb", [(1025, 24), (1064, 500), (1065, 400), (56 * 152, 39), (SHORT, 100), (SHORT + 1, 100),
                                      (248 * 300 - 1, 383), (LONG, 7), (LONG + 1, 39), (LONG + 1, 40), (300001, 385),
                                      (262144, 1000), ((1 << 21) - 5, 41)])
def test_tiles(oracle, total, nb):
    import torch
    import natural_number_gb300 as nn
    na = total - nb
    ones = np.full(na, 2**64 - 1, dtype=np.uint64)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        ctx = nn.Context(0)
        out = torch.zeros(total, dtype=torch.uint64, device="cuda")
        x, y = torch.empty(na, dtype=torch.uint64, device="cuda"), torch.empty(nb, dtype=torch.uint64, device="cuda")
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):  # a new context's words
            ctx.mul_base_device(out, x, y)
        for a, b in ((limbs(na, na), limbs(nb, nb)), (ones, np.full(nb, 2**64 - 1, dtype=np.uint64))):
            x.copy_(to_dev(a))
            y.copy_(to_dev(b))
            want = oracle.mul(a, b)
            for run in (graph.replay, lambda: ctx.mul_base_device(out, x, y), lambda: ctx.mul_base_device(out, y, x)):
                out.view(torch.int64).zero_()
                run()
                stream.synchronize()
                got = to_host(out)
                assert np.array_equal(got[: want.size], want) and not got[want.size:].any()
        ctx.close()
