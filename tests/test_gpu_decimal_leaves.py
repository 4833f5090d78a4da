"""Decimal digits on the GPU where the leaf kernel's shapes change: one to
sixteen warps a node, one limb a lane or several, first nodes shorter than the
others, runs of zero and of nine groups."""
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
sys.set_int_max_str_digits(0)


@pytest.fixture(scope="module")
def ctx():
    import natural_number_gb300 as nn
    c = nn.Context(0)
    yield c
    c.close()


def limbs_of(x):
    n = max(1, -(-x.bit_length() // 64))
    return np.frombuffer(x.to_bytes(8 * n, "little"), dtype=np.uint64).copy()


@pytest.mark.parametrize("host_below", [16, 128, 256, 1000, 4000])
@pytest.mark.parametrize("n", [2, 31, 130, 700, 1031, 9000])
def test_digits(ctx, n, host_below):
    rng = np.random.default_rng(n + host_below)
    values = [int.from_bytes(rng.integers(0, 2**64, n, dtype=np.uint64).tobytes(), "little") | 1 << (64 * n - 1),
              (1 << 64 * n) - 1, 10 ** (19 * n), 10 ** (19 * n) - 1, 10 ** (10 * n) + 7]
    for x in values:
        assert ctx.to_dec_levels(limbs_of(x), host_below) == str(x)
