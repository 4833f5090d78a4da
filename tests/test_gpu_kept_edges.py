"""Kept transforms where their calls could go wrong: residues into a buffer that
starts at an odd limb."""
import numpy as np
import pytest

from gpu_util import P, empty_dev, to_dev, to_host
from natural_number_gb300.synth import limbs

pytestmark = pytest.mark.gpu


def same_residues(got, want, s):
    got, want = got.reshape(3, 1 << s), want.reshape(3, 1 << s)
    return all(np.array_equal(got[i] % np.uint64(P[i]), want[i] % np.uint64(P[i])) for i in range(3))


@pytest.mark.parametrize("s", [2, 3, 4, 5, 11, 12, 13, 17, 21])
def test_residues_at_an_odd_limb(oracle, s):
    import natural_number_gb300 as nn
    n = (1 << s) // 2 + 1
    a = limbs(s, n)
    ctx = nn.Context(0)
    t = ctx.transform().forward(to_dev(a), s)
    buf = empty_dev((3 << s) + 3)
    t.residues(buf[1:])
    ctx.synchronize()
    got = to_host(buf)
    assert same_residues(got[1:-2], oracle.ntt_forward(a, s), s)
    assert got[0] == 0 and not got[-2:].any()
    ctx.close()
