"""Batches at every length of the contiguous pass that a scale can have, and with
items of one tile and of as many as fit, against the oracle: products of two and
three passes, a square, a split one, one-pass ones and a base case beside each
other."""
import numpy as np
import pytest

from gpu_util import empty_dev, to_dev, to_host
from natural_number_gb300.synth import limbs

pytestmark = pytest.mark.gpu


def _sizes(s):
    half = 1 << (s - 1)
    return [(half, half + 1), (half // 2 + 1, half // 2 + 9), (half - 1, half - 1), (half + 5, 130), (700, 900), (9, 5)]


@pytest.mark.parametrize("s", [13, 14, 15, 17, 19, 22])
def test_last_pass_lengths_and_item_sizes(oracle, s):
    import natural_number_gb300 as nn
    sizes = _sizes(s)
    square = [0, 0, 1, 0, 0, 0]
    ha = [limbs(5 * k + 1, x) for k, (x, _) in enumerate(sizes)]
    hb = [ha[k] if square[k] else limbs(5 * k + 2, y) for k, (_, y) in enumerate(sizes)]
    want = [oracle.mul(x, y) for x, y in zip(ha, hb)]
    a = [to_dev(x) for x in ha]
    b = [a[k] if square[k] else to_dev(x) for k, x in enumerate(hb)]
    ctx = nn.Context(0)
    ctx.set_tunable("batch_solo_scale", 0)
    levels = [r for r in range(5, 10) if 4 <= s - 3 - r <= 9] or [0]
    for r_last in levels:
        for words in (1, 8192, 1 << 20):
            ctx.set_tunable("batch_r_last@%d" % s, r_last)
            ctx.set_tunable("batch_item_words", words)
            outs = [empty_dev(x + y) for x, y in sizes]
            plan = ctx.batch([x for x, _ in sizes], [y for _, y in sizes], square)
            plan.run(list(zip(a, b)), outs)
            ctx.synchronize()
            for k, w in enumerate(want):
                got = to_host(outs[k])
                assert np.array_equal(got[: w.size], w) and not got[w.size:].any(), (r_last, words, k)
            plan.close()
    ctx.close()
