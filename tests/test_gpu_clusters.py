"""Base-case products and scans of one cluster on the GPU, at the edges of their
rules: one limb, ends of 64-position tiles and of the sixteen-CTA cluster, the
longest operand it takes, limbs of all ones (a carry through every tile)."""
import numpy as np
import pytest

from gpu_util import to_dev, to_host
from natural_number_gb300.synth import limbs

pytestmark = pytest.mark.gpu

ONES = np.uint64(2**64 - 1)


@pytest.fixture(scope="module")
def ctx():
    import natural_number_gb300 as nn
    c = nn.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("na,nb", [(1, 1), (63, 1), (33, 31), (33, 32), (64, 64), (65, 63), (65, 64), (640, 383),
                                   (640, 384), (641, 384), (640, 385), (1023, 1), (1024, 1), (512, 512),
                                   (700, 345), (2000, 96), (2049, 2040)])
def test_short_products(ctx, oracle, na, nb):
    import torch
    for fill in (False, True):
        a, b = limbs(na, na), limbs(nb + 7, nb)
        if fill:
            a[:], b[:] = ONES, ONES
        for swap in (False, True):
            x, y = (b, a) if swap else (a, b)
            out = torch.empty(na + nb + 1, dtype=torch.uint64, device="cuda")[1:]
            ctx.mul_device(out, to_dev(x), to_dev(y))
            ctx.synchronize()
            got, want = to_host(out), oracle.mul(x, y)
            assert np.array_equal(got[: want.size], want) and not got[want.size:].any()
