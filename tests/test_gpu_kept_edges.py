"""Kept transforms where their calls could go wrong: residues into a buffer that
starts at an odd limb, and a budget that holds the transforms alone."""
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


@pytest.mark.parametrize("s", [4, 5, 12, 13, 17, 20])
def test_three_factors_where_only_the_transforms_fit(oracle, s):
    """A budget that the transforms fill: products of three factors and residues
    run as they do with memory to spare, and every transform stays what it was."""
    import natural_number_gb300 as nn
    n = max((1 << s) // 4 - 1, 1)
    v = [limbs(40 * s + k, n) >> np.uint64(16) for k in range(3)]  # 48 bits: < 2^185 in all
    dev = [to_dev(x) for x in v]
    ctx = nn.Context(0, hbm_budget=5 * (24 << s))
    t = [ctx.transform() for _ in range(5)]
    out, res = empty_dev(3 * n), empty_dev((3 << s) + 1)

    def check(x, want):
        x.inverse_save(out, 3 * n)
        ctx.synchronize()
        got = to_host(out)
        k = min(want.size, got.size)
        assert np.array_equal(got[:k], want[:k]) and not got[k:].any() and not want[k:].any()

    def check_residues(x, want, at):
        x.residues(res[at:at + (3 << s)])
        ctx.synchronize()
        assert same_residues(to_host(res)[at:at + (3 << s)], oracle.ntt_forward(want, s), s)

    for i in range(3):
        t[i].forward(dev[i], s)
    t[3].pointwise(t[0], t[1])
    t[4].pointwise(t[0], t[1])
    check_residues(t[2], v[2], 0)  # through the buffer alone
    two = oracle.mul(v[0], v[1])
    t[4].pointwise(t[3], t[2])
    check(t[4], oracle.mul(two, v[2]))
    check_residues(t[2], v[2], 1)
    check_residues(t[1], v[1], 1)  # turns it over
    t[4].pointwise(t[0], t[1])  # one with the reference's words, one without
    check(t[4], two)
    t[4].pointwise(t[1], t[1])
    check(t[4], oracle.sqr(v[1]))
    t[2].pointwise(t[2], t[0])
    check(t[2], oracle.mul(v[2], v[0]))
    check(t[0], v[0])
    ctx.close()
