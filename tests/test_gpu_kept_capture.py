"""Kept transforms captured into a graph: turned back alone, as residues and as
a factor beside a product.  A replay sees the operands' new limbs, whatever the
context uploaded through its page-locked ring in between, and a transform goes
back in place, without memory."""
import numpy as np
import pytest

from gpu_util import P, empty_dev, to_dev, to_host
from natural_number_gb300.synth import limbs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s", [4, 5, 11, 12, 13, 17])
def test_replays_follow_the_operands(oracle, s):
    import torch
    import natural_number_gb300 as nn
    L, n = 1 << s, max((1 << s) // 4 - 1, 1)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        ctx = nn.Context(0)
        x = [empty_dev(n) for _ in range(3)]
        alone, prod, res = empty_dev(n + 1), empty_dev(3 * n), empty_dev(3 * L)
        t = [ctx.transform() for _ in range(5)]

        def work():
            for i in range(3):
                t[i].forward(x[i], s)
            t[3].pointwise(t[0], t[1])
            t[4].pointwise(t[3], t[2])  # three factors
            t[2].residues(res)
            t[4].inverse_save(prod, 3 * n)
            t[0].inverse_save(alone, n + 1)

        def fill(seed):
            v = [limbs(seed + k, n) >> np.uint64(16) for k in range(3)]  # 48 bits: < 2^185 in all
            for d, h in zip(x, v):
                d.copy_(to_dev(h))
            return v

        def check(v):
            stream.synchronize()
            got = to_host(alone)
            assert np.array_equal(got[:n], v[0]) and got[n] == 0
            want, got = oracle.mul(oracle.mul(v[0], v[1]), v[2]), to_host(prod)
            k = min(want.size, got.size)
            assert np.array_equal(got[:k], want[:k]) and not got[k:].any() and not want[k:].any()
            r, w = to_host(res).reshape(3, L), oracle.ntt_forward(v[2], s).reshape(3, L)
            for i in range(3):
                assert np.array_equal(r[i] % np.uint64(P[i]), w[i] % np.uint64(P[i]))

        v = fill(s)
        work()
        check(v)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            work()
        pool, out, count = to_dev(limbs(99, 16)), empty_dev(16 * 3000), 3000
        jobs = (nn.MulJob * count)()
        for j in range(count):
            jobs[j] = nn.MulJob(pool.data_ptr(), 9, pool.data_ptr() + 72, 7, out.data_ptr() + 128 * j)
        plan = ctx.batch([9] * count, [7] * count)
        for k in range(3):
            v = fill(100 * s + 10 * k)
            for _ in range(60):  # other uploads take the ring's bytes in turn
                ctx._check(nn.lib().nn_batch_launch(ctx.h, plan.h, jobs), "batch")
            ctx.synchronize()
            graph.replay()
            check(v)
        ctx.close()


def test_turning_back_takes_no_memory():
    import natural_number_gb300 as nn
    s, n = 16, 1 << 15
    a = limbs(5, n)
    ctx = nn.Context(0, hbm_budget=24 << s)
    t = ctx.transform().forward(to_dev(a), s)
    out = empty_dev(n + 1)
    t.inverse_save(out, n + 1)
    ctx.synchronize()
    got = to_host(out)
    assert np.array_equal(got[:n], a) and got[n] == 0
    ctx.close()
