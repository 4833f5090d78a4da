"""The batched differences of the decimal split at lengths of one CTA a job:
one step of 1024 limbs or many, and borrows that run through all of them
(values next to powers of the split's bases)."""
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
sys.set_int_max_str_digits(0)


@pytest.mark.parametrize("n", [1100, 2300, 4200, 40000])
def test_digits_next_to_powers(n):
    import natural_number_gb300 as nn
    ctx = nn.Context(0)
    rng = np.random.default_rng(n)
    digits = 18 * (1 << (int(n * 64 / 59.8).bit_length() - 1))  # a split base of the largest level
    cases = {"1" + "0" * digits, "9" * digits, "1" + "0" * (digits - 1) + "1",
             "".join(map(str, rng.integers(1, 10, digits + 5)))}
    for text in cases:
        x = int(text)
        a = np.frombuffer(x.to_bytes((x.bit_length() + 63) // 64 * 8, "little"), dtype=np.uint64).copy()
        assert ctx.to_dec_levels(a) == text
    ctx.close()
