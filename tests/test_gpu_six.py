"""The six-prime products on the GPU at the edges of their shapes: every
transform scale with the fewest and the most coefficients it holds (half and
whole first-pass tiles, one, two and three passes, blocks of 8 to 64
coefficients), pieces of an unbalanced operand, operands at odd 8-byte
addresses, limbs of all ones (the largest coefficients)."""
import numpy as np
import pytest

from gpu_util import mod_checks, to_dev, to_host
from natural_number_gb300.synth import limbs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import natural_number_gb300 as nn
    c = nn.Context(0)
    yield c
    c.close()


def product(ctx, a, b):
    import torch
    out = torch.empty(a.numel() + b.numel(), dtype=torch.uint64, device="cuda")
    ctx.mul_device(out, a, b)
    ctx.synchronize()
    return out


def check_mod(ctx, a, b, out):
    ma, mb, mp = mod_checks(to_host(a)), mod_checks(to_host(b)), mod_checks(to_host(out))
    assert mp[0] == ma[0] * mb[0] % (2**64 - 1) and mp[1] == ma[1] * mb[1] % (2**64 + 1)


@pytest.mark.parametrize("s", range(10, 20))
def test_every_scale_vs_oracle(ctx, oracle, s):
    half = 1 << (s - 1)
    for na, nb in [(half // 2 + 1, half // 2 + 1), (half, half + 1), (half + 1, half), (half - 3, half - 130)]:
        a, b = limbs(s * 11 + na, na), limbs(s * 13 + nb, nb)
        got = to_host(product(ctx, to_dev(a), to_dev(b)))
        want = oracle.mul(a, b)
        assert np.array_equal(got[: want.size], want) and not got[want.size:].any()
        import torch
        sq = torch.empty(2 * na, dtype=torch.uint64, device="cuda")
        ctx.sqr_device(sq, to_dev(a))
        got, want = to_host(sq), oracle.sqr(a)
        assert np.array_equal(got[: want.size], want) and not got[want.size:].any()


@pytest.mark.parametrize("s", [6, 9, 10, 12, 13, 14, 17, 18, 19, 22])
def test_truncated_transforms_vs_oracle(ctx, oracle, s):
    """Products that end at, just below and just above each eighth of the
    transform, one at a time and in a batch (which takes the short ones too)."""
    import torch
    L = 1 << s
    sizes = []
    for k in (5, 6, 7):
        for length in (k * L // 8 - 1, k * L // 8, k * L // 8 + 1):
            na = length // 2 + 1 + (length // 16 if k == 6 else 0)
            sizes.append((na, length + 1 - na))
    a_list = [limbs(s + k, na) for k, (na, _) in enumerate(sizes)]
    b_list = [limbs(s + 50 + k, nb) for k, (_, nb) in enumerate(sizes)]
    da, db = [to_dev(a) for a in a_list], [to_dev(b) for b in b_list]
    outs = [torch.empty(na + nb, dtype=torch.uint64, device="cuda") for na, nb in sizes]
    old = {k: ctx.get_tunable(k) for k in ("batch_ntt_min", "batch_school_balanced")}
    try:
        ctx.set_tunable("batch_ntt_min", 1)
        ctx.set_tunable("batch_school_balanced", 0)
        ctx.batch([x for x, _ in sizes], [y for _, y in sizes]).run(list(zip(da, db)), outs)
        ctx.synchronize()
    finally:
        for k, v in old.items():
            ctx.set_tunable(k, v)
    for k in range(len(sizes)):
        want = oracle.mul(a_list[k], b_list[k])
        for got in (to_host(product(ctx, da[k], db[k])), to_host(outs[k])):
            assert np.array_equal(got[: want.size], want) and not got[want.size:].any(), sizes[k]


@pytest.mark.parametrize("s", [20, 21, 22, 23, 24, 25, 26, 27, 28])
def test_long_scales_by_residues(ctx, s):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(s)
    half = 1 << (s - 1)
    for na, nb in [(half // 2 + 1, half // 2 + 7), (half, half + 1)]:
        a, b = (torch.randint(-(2**63), 2**63 - 1, (n,), dtype=torch.int64, device="cuda", generator=g)
                .view(torch.uint64) for n in (na, nb))
        check_mod(ctx, a, b, product(ctx, a, b))
        if s % 2 == 0:
            out = torch.empty(2 * na, dtype=torch.uint64, device="cuda")
            ctx.sqr_device(out, a)
            ctx.synchronize()
            check_mod(ctx, a, a, out)


@pytest.mark.parametrize("na,nb", [(5000, 384), (70001, 400), (300007, 2049), (1 << 20, 5003), (40000, 12001)])
def test_pieces_vs_oracle(ctx, oracle, na, nb):
    a, b = limbs(na, na), limbs(nb, nb)
    a[: na // 2] = np.uint64(0xFFFFFFFFFFFFFFFF)  # largest overlaps
    b[:] = np.uint64(0xFFFFFFFFFFFFFFFF)
    for x, y in ((a, b), (b, a)):
        got, want = to_host(product(ctx, to_dev(x), to_dev(y))), oracle.mul(a, b)
        assert np.array_equal(got[: want.size], want) and not got[want.size:].any()


@pytest.mark.parametrize("n", [600, 5000, 1 << 17, (1 << 24) + 5])
def test_odd_addresses_and_all_ones(ctx, n):
    import torch
    a = torch.full((n + 3,), -1, dtype=torch.int64, device="cuda").view(torch.uint64)
    out = torch.empty(2 * n + 1, dtype=torch.uint64, device="cuda")
    for oa, ob, oo in ((0, 0, 0), (1, 2, 1), (3, 1, 0)):
        ctx.mul_device(out[oo:oo + 2 * n], a[oa:oa + n], a[ob:ob + n])
        ctx.synchronize()
        got = to_host(out[oo:oo + 2 * n])  # (B^n - 1)^2 = B^2n - 2 B^n + 1
        ones = np.uint64(0xFFFFFFFFFFFFFFFF)
        assert got[0] == 1 and not got[1:n].any() and got[n] == ones - np.uint64(1) and (got[n + 1:] == ones).all()


@pytest.mark.parametrize("s", [4, 5, 8, 12, 13, 17, 21, 22, 26])
def test_kept_transforms(ctx, oracle, s):
    """A transform kept and multiplied, squared and turned back alone, in normal
    and wrap mode; residues of a product's transform, and a product of three,
    whose factors leave the six primes for the three-prime words."""
    from gpu_util import P, empty_dev
    L = 1 << s
    na, nb = max(L // 2 - 3, 2), max(L // 2 - 1, 2)
    a, b = limbs(s + 1, na), limbs(s + 2, nb)
    ta, tb = ctx.transform().forward(to_dev(a), s), ctx.transform().forward(to_dev(b), s)
    out = empty_dev(L + 2)
    prod = ctx.transform().pointwise(ta, tb)
    for _ in range(2):  # a product's residues can be saved again
        w = prod.inverse_save(out, na + nb)
        ctx.synchronize()
        if s <= 22:
            want = oracle.mul(a, b)
            got = to_host(out, w)
            assert np.array_equal(got[: want.size], want) and not got[want.size:].any()
        else:
            check_mod(ctx, to_dev(a), to_dev(b), out[: na + nb])
    if s > 17:
        return
    sq = ctx.transform().pointwise(ta, ta)
    sq.inverse_save(out, 2 * na)
    want = oracle.sqr(a)
    assert np.array_equal(to_host(out, 2 * na)[: want.size], want)
    full = limbs(s + 3, L)  # wraps modulo B^L - 1
    tf = ctx.transform().forward(to_dev(full), s)
    assert ctx.transform().pointwise(tf, tb).inverse_save(out, L + 2) == L
    assert np.array_equal(to_host(out, L), oracle.ntt_mul_raw(full, b, s, L + 2))
    alone = ctx.transform().forward(to_dev(a), s)
    alone.inverse_save(out, na + 1)
    got = to_host(out, na + 1)
    assert np.array_equal(got[:na], a) and got[na] == 0
    res3, want3 = empty_dev(3 * L), empty_dev(3 * L)
    one = ctx.transform().forward(to_dev(np.array([1], dtype=np.uint64)), s)
    ctx.transform().pointwise(ta, one).residues(res3)
    ta.residues(want3)
    r, v = to_host(res3).reshape(3, L), to_host(want3).reshape(3, L)
    for i in range(3):
        assert np.array_equal(r[i] % np.uint64(P[i]), v[i] % np.uint64(P[i]))
    small = [limbs(s + 7 + k, max(L // 4 - 2, 1)) >> np.uint64(16) for k in range(3)]  # 48-bit limbs: < 2^185 in all
    t3 = [ctx.transform().forward(to_dev(x), s) for x in small]
    t3[2].pointwise(ctx.transform().pointwise(t3[0], t3[1]), t3[2])
    n = 3 * small[0].size
    t3[2].inverse_save(out, n)
    want = oracle.mul(oracle.mul(small[0], small[1]), small[2])
    got = to_host(out, n)
    k = min(n, want.size)
    assert np.array_equal(got[:k], want[:k]) and not got[k:].any() and not want[k:].any()
