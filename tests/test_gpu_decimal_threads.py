"""Decimal conversions in two threads whose leaves take different amounts of
shared memory, each with its own context."""
import threading

import numpy as np
import pytest

from natural_number_gb300.synth import limbs

pytestmark = pytest.mark.gpu


def test_leaves_of_different_sizes_in_two_threads():
    import natural_number_gb300 as nn
    a = limbs(11, 8000)
    ctx = [nn.Context(0, use_torch_stream=False) for _ in range(2)]
    below = (4000, 3000)  # leaves of up to 7654 and 3827 limbs: 61 and 37 KB
    want = [c.to_dec_levels(a, b) for c, b in zip(ctx, below)]  # powers and tables are there
    assert want[0] == want[1]
    failed = []

    def convert(c, b):
        try:
            for _ in range(60):
                if c.to_dec_levels(a, b) != want[0]:
                    raise AssertionError("digits")
        except Exception as e:  # noqa: BLE001
            failed.append(e)

    threads = [threading.Thread(target=convert, args=x) for x in zip(ctx, below)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for c in ctx:
        c.close()
    assert not failed
