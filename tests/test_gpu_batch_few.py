"""Batches of a few products: the rule that gives short ones a common scale and
leaves longer ones whole, against the oracle and against every product by its own
plan; unbalanced products alone keep their pieces."""
import numpy as np
import pytest

from gpu_util import empty_dev, to_dev, to_host
from natural_number_gb300.synth import limbs

pytestmark = pytest.mark.gpu


def _run(ctx, sizes, a, b, few):
    ctx.set_tunable("batch_few", few)
    plan = ctx.batch([x for x, _ in sizes], [y for _, y in sizes])
    outs = [empty_dev(x + y) for x, y in sizes]
    plan.run(list(zip(a, b)), outs)
    ctx.synchronize()
    got, items = [to_host(o) for o in outs], plan.items
    plan.close()
    return got, items


@pytest.mark.parametrize("sizes,same", [
    ([(16000, 300)] * 5, True),
    ([(8000, 70), (9000, 400), (300, 12000)], True),
    ([(8000, 70), (8000, 7900), (16000, 300)], False),  # beside a whole one of two passes
    ([(2000, 2000)] + [(200, 64)] * 40, False),
    ([(64, 64), (4095, 2), (100, 3996), (2049, 2047)], False),
    ([(600, 500)] * 153, True),  # not a few
])
def test_few(oracle, sizes, same):
    import natural_number_gb300 as nn
    ctx = nn.Context(0)
    ha = [limbs(3 * k + 1, x) for k, (x, _) in enumerate(sizes)]
    hb = [limbs(3 * k + 2, y) for k, (_, y) in enumerate(sizes)]
    a, b = [to_dev(x) for x in ha], [to_dev(x) for x in hb]
    got, items = _run(ctx, sizes, a, b, 1)
    own, own_items = _run(ctx, sizes, a, b, 0)
    for k in range(len(sizes)):
        want = oracle.mul(ha[k], hb[k])
        for g in (got[k], own[k]):
            assert np.array_equal(g[: want.size], want) and not g[want.size:].any()
    if same:
        assert items == own_items
    ctx.close()
