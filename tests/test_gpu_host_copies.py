"""Products of host operands on both sides of the line of their copies in
ranges, in page-locked and pageable memory and a mix, from odd addresses."""
import numpy as np
import pytest

from gpu_util import mod_checks
from natural_number_gb300.synth import limbs

pytestmark = pytest.mark.gpu


def _host(n, locked):
    import torch
    t = torch.empty(n + 1, dtype=torch.int64, pin_memory=bool(locked))
    return t.numpy().view(np.uint64)[1:]


@pytest.mark.parametrize("locked", [(1, 1, 1), (0, 0, 0), (1, 0, 1), (1, 1, 0), (0, 1, 1)])
@pytest.mark.parametrize("na,nb", [(700, 600), (1 << 20, 1 << 20), ((1 << 20) + 1, 1 << 20), (900001, 1500000)])
def test_host_product(na, nb, locked):
    import natural_number_gb300 as nn
    a, b, out = _host(na, locked[0]), _host(nb, locked[1]), _host(na + nb, locked[2])
    a[:], b[:] = limbs(na, na), limbs(nb + 1, nb)
    ctx = nn.Context(0)
    for _ in range(2):
        out[:] = 0
        ctx.mul(a, b, out)
        ma, mb, mp = mod_checks(a), mod_checks(b), mod_checks(out)
        assert mp[0] == ma[0] * mb[0] % (2**64 - 1) and mp[1] == ma[1] * mb[1] % (2**64 + 1)
    ctx.close()
