"""Products on both sides of each line of the base-case rule against the oracle
and the base case itself; a budget that holds no residues and a capture before
the first transform fall back to the base case."""
import numpy as np
import pytest

from gpu_util import to_dev, to_host
from natural_number_gb300.synth import limbs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import natural_number_gb300 as nn
    c = nn.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("nb", [1, 31, 32, 33, 95, 96, 97, 255, 256, 257, 383, 384])
@pytest.mark.parametrize("na", [0, 900, 929, 1024, 16383, 16384, 70001])
def test_rule(ctx, oracle, na, nb):
    import torch
    na = max(na, nb)
    for fill in (False, True):
        a, b = limbs(na + 1, na), limbs(nb + 2, nb)
        if fill:
            a[:], b[:] = np.uint64(2**64 - 1), np.uint64(2**64 - 1)
        want = oracle.mul(a, b)
        da, db = torch.empty(na + 1, dtype=torch.uint64, device="cuda")[1:], to_dev(b)  # an odd address
        da.copy_(to_dev(a))
        outs = [torch.empty(na + nb, dtype=torch.uint64, device="cuda") for _ in range(3)]
        ctx.mul_device(outs[0], da, db)
        ctx.mul_device(outs[1], db, da)
        ctx.mul_base_device(outs[2], da, db)
        ctx.synchronize()
        for o in outs:
            got = to_host(o)
            assert np.array_equal(got[: want.size], want) and not got[want.size:].any()
    if na == nb:
        sq = torch.empty(2 * na, dtype=torch.uint64, device="cuda")
        ctx.sqr_device(sq, da)
        ctx.synchronize()
        got, want = to_host(sq), oracle.sqr(a)
        assert np.array_equal(got[: want.size], want) and not got[want.size:].any()


@pytest.mark.parametrize("na,nb", [(300, 300), (5000, 100), (100000, 300)])
def test_no_room_and_capture(oracle, na, nb):
    import torch
    import natural_number_gb300 as nn
    a, b = limbs(na, na), limbs(nb + 3, nb)
    want = oracle.mul(a, b)
    da, db = to_dev(a), to_dev(b)
    out = torch.empty(na + nb, dtype=torch.uint64, device="cuda")

    def check():
        got = to_host(out)
        assert np.array_equal(got[: want.size], want) and not got[want.size:].any()
        out.view(torch.int64).zero_()

    small = nn.Context(0, hbm_budget=4096)
    small.mul_device(out, da, db)
    small.synchronize()
    check()
    small.close()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        c = nn.Context(0)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            c.mul_device(out, da, db)
        graph.replay()
        stream.synchronize()
        check()
        c.mul_device(out, da, db)  # outside the capture, with tables
        stream.synchronize()
        check()
        c.close()
