"""Chains of dependent calls on one stream: every kernel waits for the writes of
the one before it, whether that is ours, a copy or another library's kernel,
and keeps its order when a chain is captured into a graph and replayed."""
import numpy as np
import pytest

from gpu_util import to_dev, to_host
from natural_number_gb300.synth import limbs

pytestmark = pytest.mark.gpu


def chain(ctx, out, x, y, t, u):
    """out = (~x * y) squared, modulo the size of `out`."""
    import torch
    torch.bitwise_not(x.view(torch.int64), out=u.view(torch.int64))
    ctx.mul_device(t, u, y)
    ctx.sqr_device(out, t)


@pytest.mark.parametrize("n", [40, 300, 1000, 2500, 30000, 300000])
def test_chain_and_captured_chain(oracle, n):
    import torch
    import natural_number_gb300 as nn
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        ctx = nn.Context(0)
        empty = lambda k: torch.empty(k, dtype=torch.uint64, device="cuda")
        x, y, t, u, out = empty(n), empty(n), empty(2 * n), empty(n), empty(4 * n)

        def check(seed, run):
            a, b = limbs(seed, n), limbs(seed + 1, n)
            x.copy_(to_dev(a))
            y.copy_(to_dev(b))
            out.view(torch.int64).zero_()
            run()
            stream.synchronize()
            p = oracle.mul(~a, b)
            want = oracle.sqr(p)
            got = to_host(out)
            assert np.array_equal(got[: want.size], want) and not got[want.size:].any()

        for k in range(4):
            check(10 * k + n, lambda: chain(ctx, out, x, y, t, u))
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            chain(ctx, out, x, y, t, u)
        for k in range(4):
            check(100 * k + n, graph.replay)
        ctx.close()
