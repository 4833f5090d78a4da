"""A batch's first run (launch by launch), its second (which makes the graph) and
later ones, on operands that change in between; first runs of two plans of one
context on two streams."""
import numpy as np
import pytest

from gpu_util import empty_dev, to_dev, to_host
from natural_number_gb300.synth import limbs

pytestmark = pytest.mark.gpu

SIZES = [(9, 5), (100, 70), (700, 900), (3000, 200), (5000, 4999), (20000, 300), (40000, 41001), (150000, 64)]


def _same(got, want):
    return np.array_equal(got[: want.size], want) and not got[want.size:].any()


@pytest.mark.parametrize("count", [1, 3, 8, 160])
def test_runs_of_one_plan(oracle, count):
    import natural_number_gb300 as nn
    sizes = [SIZES[(5 * k) % len(SIZES)] for k in range(count)] if count <= 8 else [SIZES[k % 4] for k in range(count)]
    ctx = nn.Context(0)
    a, b = [empty_dev(x) for x, _ in sizes], [empty_dev(y) for _, y in sizes]
    outs = [[empty_dev(x + y) for x, y in sizes] for _ in range(2)]
    plan = ctx.batch([x for x, _ in sizes], [y for _, y in sizes])
    for run in range(4):
        ha = [limbs(100 * run + 2 * k, x) for k, (x, _) in enumerate(sizes)]
        hb = [limbs(100 * run + 2 * k + 1, y) for k, (_, y) in enumerate(sizes)]
        for d, h in zip(a + b, ha + hb):
            d.copy_(to_dev(h))
        o = outs[run % 2]
        plan.run(list(zip(a, b)), o)
        ctx.synchronize()
        for k in range(count):
            assert _same(to_host(o[k]), oracle.mul(ha[k], hb[k])), (run, k)
    plan.close()
    ctx.close()


def test_first_runs_on_two_streams(oracle):
    import torch
    import natural_number_gb300 as nn
    ctx = nn.Context(0)
    ctx.set_tunable("batch_solo_scale", 0)
    streams = [torch.cuda.Stream() for _ in range(2)]
    ha = [[limbs(1000 * p + 2 * k, x) for k, (x, _) in enumerate(SIZES)] for p in range(2)]
    hb = [[limbs(1000 * p + 2 * k + 1, y) for k, (_, y) in enumerate(SIZES)] for p in range(2)]
    a, b = [[to_dev(x) for x in h] for h in ha], [[to_dev(x) for x in h] for h in hb]
    outs = [[empty_dev(x + y) for x, y in SIZES] for _ in range(2)]
    torch.cuda.synchronize()
    for _ in range(5):
        plans = []
        for p in range(2):
            ctx.set_stream(streams[p].cuda_stream)
            plans.append(ctx.batch([x for x, _ in SIZES], [y for _, y in SIZES]))
            plans[p].run(list(zip(a[p], b[p])), outs[p])
        torch.cuda.synchronize()
        for p in range(2):
            ctx.set_stream(streams[p].cuda_stream)
            plans[p].close()
            for k in range(len(SIZES)):
                assert _same(to_host(outs[p][k]), oracle.mul(ha[p][k], hb[p][k])), (p, k)
                outs[p][k].view(torch.int64).zero_()
        torch.cuda.synchronize()
    ctx.set_stream(None)
    ctx.close()
