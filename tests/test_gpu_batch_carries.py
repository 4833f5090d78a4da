"""Carries between the tiles of batched products: operands of all ones, whose
products hold runs of all-ones limbs over many tiles of 2048, whole and in
pieces, next to random ones."""
import numpy as np
import pytest

from gpu_util import to_dev, to_host
from natural_number_gb300.synth import limbs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[(64, 64), (1024, 1024), (1025, 1024), (2048, 2047)],
                                   [(9000, 5000), (70000, 2000), (40000, 40000)],
                                   [(100000, 300), (5, 4096), (4096, 4097), (300000, 70)]])
def test_runs_of_ones(oracle, sizes):
    import torch
    import natural_number_gb300 as nn
    ctx = nn.Context(0)
    pairs = []
    for k, (na, nb) in enumerate(sizes):
        a, b = limbs(k + na, na), limbs(k + nb + 1, nb)
        ones = [np.full(n, 2**64 - 1, dtype=np.uint64) for n in (na, nb)]
        power = np.zeros(na, dtype=np.uint64)
        power[na // 2] = 1
        pairs += [(ones[0], ones[1]), (a, b), (ones[0], b), (power, ones[1])]
    plan = ctx.batch([x.size for x, _ in pairs], [y.size for _, y in pairs])
    dev = [(to_dev(x), to_dev(y), torch.empty(x.size + y.size, dtype=torch.uint64, device="cuda")) for x, y in pairs]
    for _ in range(2):
        plan.run([(x, y) for x, y, _ in dev], [o for _, _, o in dev])
        ctx.synchronize()
        for (x, y), (_, _, o) in zip(pairs, dev):
            got, want = to_host(o), oracle.mul(x, y)
            assert np.array_equal(got[: want.size], want) and not got[want.size:].any()
    plan.close()
    ctx.close()
