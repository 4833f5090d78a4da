"""The six-prime product (natural_number_gb300/csrc/six_tiles.cuh, six.cu,
scan_tiles.cuh), restated in Python and checked on the CPU: the tiles' index
arithmetic, the lazy ranges at their worst, the CRT's quotient at the ends of
its range, and whole products (tree, blocks, scale factors) against Python's
integers."""
import math
import random

import pytest

MUL = [25, 27, 33, 37, 39, 40]
P = [(m << 22) | 1 for m in MUL]
M = math.prod(P)
LIMIT = 1 << 31


def groups(R):
    if R == 4:
        return [(0, 3), (3, 1)]
    n, left, out, l = (R + 2) // 3, R, [], 0
    for i in range(n):
        k = -(-left // (n - i))
        out.append((l, k))
        l += k
        left -= k
    return out


def at(C, leaf, row):
    if not leaf:
        return row * C
    return row * C + (row >> 3) * C if C == 8 else row * (C + (4 if C == 16 else C // 8))


def tile_words(C, leaf, R):
    if not leaf:
        return C << R
    return (C << R) + (((1 << R) + 7) // 8) * C if C == 8 else (C + (4 if C == 16 else C // 8)) << R


def col_width(R):
    return 32 if R >= 7 else 4096 >> R


@pytest.mark.parametrize("C,leaf,R", [(8, True, r) for r in range(1, 10)] + [
    (16, True, 8), (32, True, 7), (64, True, 6), (128, True, 5), (256, True, 4), (512, True, 4)] + [
    (col_width(r), False, r) for r in range(4, 10)])
@pytest.mark.parametrize("V", [1, 2, 4])
def test_units_cover_the_tile(C, leaf, R, V):
    for l, K in groups(R):
        nsub, seen = R - l - K, set()
        for i in range((C // V) << (R - K)):
            col, v = (i % (C // V)) * V, i // (C // V)
            rb = v >> nsub
            row0 = (rb << (nsub + K)) + (v & ((1 << nsub) - 1))
            for m in range(1 << K):
                row = row0 + (m << nsub)
                word = at(C, leaf, row0) + col + at(C, leaf, m << nsub)
                assert word == at(C, leaf, row) + col and word % V == 0 and word + V <= tile_words(C, leaf, R)
                seen.add((row, col))
        assert len(seen) == (C // V) << R


def test_primes():
    for i, p in enumerate(P):
        assert all(p % d for d in range(3, 13000, 2)) and (p - 1) % (1 << 22) == 0
        assert (p * (1 - (MUL[i] << 22))) % (1 << 32) == 1
    assert M.bit_length() == 163 and M > 4 << 160  # two overlapping pieces of 2^31 limbs: below M / 4


@pytest.mark.parametrize("p", P)
def test_lazy_ranges(p):
    step = lambda y: 0.5 + y * p / 2**33  # noqa: E731  magnitude of a product, in p
    lim = LIMIT / p
    x = 1.0  # limbs
    for _ in range(18):
        x += step(x)
    assert x < lim
    x = step(lim)  # reduced at the last pass's start
    assert x <= 0.75
    for _ in range(9):
        x += step(x)
    assert x < lim and step(x) <= 0.75  # reduced again before the blocks' products
    assert 8 * (0.75 * p) ** 2 / 2**32 + p / 2 <= 1.5 * p  # an 8-block's product after its Montgomery step
    for m in (16, 32, 64, 128, 256, 512):  # longer blocks: 64-bit sums, then reduced
        assert m * (0.75 * p) ** 2 < 2**63 and m * (0.75 * p) ** 2 / 2**32 + p / 2 + 0.75 * p < LIMIT
    for K in (1, 2, 3):  # inverse groups from 1.5 p
        bound = [1.5] * (1 << K)
        for lv in range(K - 1, -1, -1):
            half = (1 << K) >> (lv + 1)
            for g in range(1 << lv):
                for m in range(half):
                    i, j = g * 2 * half + m, g * 2 * half + m + half
                    s = bound[i] + bound[j]
                    assert s < lim
                    bound[i], bound[j] = s, step(s)
        assert all(b <= 1.5 for b in bound[(2 if K == 3 else 1):])


def companion(w, p):
    n, h = w << 32, p // 2
    q = (abs(n) + h) // p
    return q if n >= 0 else -q


def mul_mod(y, w, p):
    q = (y * companion(w, p) + (1 << 31)) >> 32
    r = y * w - q * p
    assert abs(r) <= (0.5 + abs(y) / 2**33) * p + 1
    return r


def center(w, p):
    w %= p
    return w - p if w > p // 2 else w


def crt(y):
    cols, frac = [0] * 6, 1 << 24
    for i, p in enumerate(P):
        t = y[i] + 2 * p
        assert 0 < t < 4 * p
        frac += (t >> 12) * (((1 << 39) + p // 2) // p)
        m = M // p
        for j in range(5):
            cols[j] += t * ((m >> (32 * j)) & 0xffffffff)
        assert m >> 160 == 0
    assert frac < 1 << 32 and max(cols) < (1 << 64) - (1 << 37)
    neg = (1 << 192) - M
    v = sum(c << (32 * j) for j, c in enumerate(cols)) + (frac >> 27) * neg
    return v % (1 << 192)


def test_crt_quotient_over_its_range():
    rng = random.Random(3)
    inv = [pow(M // p, -1, p) for p in P]
    values = [0, 1, 2, (1 << 160) - 1, 1 << 160, (1 << 128) - 1] + [rng.randrange(1 << 160) for _ in range(2000)]
    values += [rng.randrange(1 << rng.randrange(1, 161)) for _ in range(2000)]
    for v in values:
        base = [center(v * k, p) for k, p in zip(inv, P)]
        for shift in ([0] * 6, [1] * 6, [-1] * 6, [rng.choice((-1, 0, 1)) for _ in P]):  # up to 1.5 p
            assert crt([r + d * p for r, d, p in zip(base, shift, P)]) == v


@pytest.mark.parametrize("p", P)
@pytest.mark.parametrize("k8", [5, 6, 7])
def test_truncated_last_group(p, k8):
    """Rows y_b = P(c_b) of a polynomial of k8 coefficients at the first k8 of
    the eight points, to 16 times its coefficients; every intermediate at its
    worst stays in 32 bits."""
    rng = random.Random(p + k8)
    g = root(p)
    i, w = pow(g, 1 << 20, p), pow(g, 1 << 19, p)
    h = i * w % p
    points = [1, p - 1, i, p - i, w, p - w, h, p - h]
    a = [rng.randrange(p) for _ in range(k8)]
    y = [sum(v * pow(points[b], j, p) for j, v in enumerate(a)) for b in range(k8)] + [0] * (8 - k8)
    ii, wi = pow(i, -1, p), pow(w, -1, p)
    u0, u2 = y[0] + y[1] + y[2] + y[3], y[0] + y[1] - y[2] - y[3]
    d1 = (y[2] - y[3]) * ii
    u1, u3 = y[0] - y[1] + d1, y[0] - y[1] - d1
    out = [0] * 8
    if k8 == 5:
        d = 4 * y[4] - w * u1 - i * u2 - h * u3
        out = [2 * (u0 + d), 4 * u1, 4 * u2, 4 * u3, 2 * (u0 - d)]
    else:
        v0, v1 = y[4] + y[5], (y[4] - y[5]) * wi
        e = 2 * v1 - i * u3
        out[1], out[5], out[3] = 2 * (u1 + e), 2 * (u1 - e), 4 * u3
        if k8 == 6:
            d = 2 * v0 - i * u2
            out[0], out[4], out[2] = 2 * (u0 + d), 2 * (u0 - d), 4 * u2
        else:
            f = 4 * y[6] - h * e - w * u3
            q = (2 * v0 - f) * i
            out[0], out[4] = 2 * u0 + 2 * v0 + f, 2 * u0 - 2 * v0 - f
            out[2], out[6] = 2 * u2 - q, 2 * u2 + q
    assert [v % p for v in out[:k8]] == [16 * v % p for v in a]
    step = lambda x: 0.5 + x * p / 2**33  # noqa: E731  a product or a reduction, in p; rows come in below 1.5 p
    u, v = step(6.0), step(3.0)
    d5, d6 = 4 * step(1.5) + 3 * step(u), 2 * v + step(u)
    f7 = 4 * step(1.5) + step(d6) + step(u)
    assert max(2 * (u + d5), 2 * (u + d6), 2 * u + 2 * v + f7, 4 * u, 2 * v + f7) < LIMIT / p  # then scaled, to 0.75 p


def root(p):
    a = 2
    while True:
        g = pow(a, (p - 1) >> 22, p)
        if pow(g, 1 << 21, p) == p - 1:
            return g
        a += 1


@pytest.mark.parametrize("s,T,na,nb", [(4, 1, 9, 8), (6, 3, 33, 30), (7, 4, 100, 29), (8, 5, 255, 2), (8, 3, 130, 127),
                                       (9, 4, 256, 257), (9, 3, 300, 200)])
def test_products(s, T, na, nb):
    """Tree of T levels from limbs times 2^-32, blocks of 2^(s-T) coefficients, inverse, CRT."""
    rng = random.Random(s * 100 + T)
    A, B = [[rng.getrandbits(64) for _ in range(n)] for n in (na, nb)]
    L, m = 1 << s, 1 << (s - T)
    res = []
    for p in P:
        g, r32 = root(p), pow(2, -32, p)
        W = [1] * (1 << T)
        for b in range(1 << T):
            for t in range(T):
                if (b >> t) & 1:
                    W[b] = W[b] * pow(g, 1 << (20 - t), p) % p
        cur = []
        for X in (A, B):
            x = [v * r32 % p for v in X] + [0] * (L - len(X))
            for lv in range(T):
                h = L >> (lv + 1)
                for b in range(1 << lv):
                    for i in range(h):
                        u, v = x[2 * b * h + i], x[2 * b * h + h + i] * W[b] % p
                        x[2 * b * h + i], x[2 * b * h + h + i] = (u + v) % p, (u - v) % p
            cur.append(x)
        a, b = cur
        o = [0] * L
        for blk in range(1 << T):
            c = W[blk >> 1] if blk % 2 == 0 else -W[blk >> 1]
            for i in range(m):
                for j in range(m):
                    v = a[blk * m + i] * b[blk * m + j] * r32
                    o[blk * m + (i + j) % m] += v * c if i + j >= m else v
        o = [v % p for v in o]
        for lv in range(T - 1, -1, -1):
            h = L >> (lv + 1)
            for b in range(1 << lv):
                wi = pow(W[b], -1, p)
                for i in range(h):
                    u, v = o[2 * b * h + i], o[2 * b * h + h + i]
                    o[2 * b * h + i], o[2 * b * h + h + i] = (u + v) % p, (u - v) * wi % p
        res.append(o)
    scale = [pow(2, 96 - T, p) * pow(M // p, -1, p) for p in P]
    total = sum(crt([mul_mod(center(res[i][k], P[i]), center(scale[i], P[i]), P[i]) for i in range(6)]) << (64 * k)
                for k in range(na + nb - 1))
    val = lambda X: sum(v << (64 * i) for i, v in enumerate(X))  # noqa: E731
    assert total == val(A) * val(B)
