"""Products written over their own operands: device buffers that hold the longer
operand, the shorter one or both of a square, from the buffer's first limb or a
later one, on every route of nn_mul."""
import numpy as np
import pytest

from gpu_util import to_dev, to_host
from natural_number_gb300.synth import limbs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("na,nb", [(3, 2), (64, 48), (900, 100), (1000, 25), (5000, 20), (60000, 30), (131072, 16),
                                   (300000, 31), (300, 300), (5000, 200), (1500, 1201), (40000, 30001), (300000, 2500)])
def test_product_over_its_operands(oracle, na, nb):
    import torch
    import natural_number_gb300 as nn
    ctx = nn.Context(0)
    a, b = limbs(na, na), limbs(nb + 1, nb)
    want, square, based = oracle.mul(a, b), oracle.sqr(b), na + nb < 200000
    total = na + nb
    for at in {0, 1, nb // 2, nb}:
        for which in ("a", "b"):
            x, other, n = (a, b, na) if which == "a" else (b, a, nb)
            for call in (ctx.mul_device, ctx.mul_base_device) if based else (ctx.mul_device,):
                buf = torch.zeros(total, dtype=torch.uint64, device="cuda")
                buf[at:at + n].copy_(to_dev(x))
                call(buf, buf[at:at + n], to_dev(other))
                ctx.synchronize()
                got = to_host(buf)
                assert np.array_equal(got[: want.size], want) and not got[want.size:].any(), (at, which)
    buf = torch.zeros(2 * nb, dtype=torch.uint64, device="cuda")
    buf[:nb].copy_(to_dev(b))
    ctx.sqr_device(buf, buf[:nb])
    ctx.synchronize()
    got = to_host(buf)
    assert np.array_equal(got[: square.size], square) and not got[square.size:].any()
    ctx.close()
