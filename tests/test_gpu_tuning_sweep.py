"""The batch sweep of the tuner settles every batch tunable that the package's
file sets, so that a file it writes leaves none at a default."""
import json

import pytest

pytestmark = pytest.mark.gpu


def test_batch_sweep_covers_the_package_file():
    import natural_number_gb300 as nn
    from natural_number_gb300 import autotune
    with open(autotune.TUNING) as f:
        packaged = json.load(f)["tunables"]
    ctx = nn.Context(0)
    best, log = autotune.tune_batch(ctx, 48)
    ctx.close()
    assert {k for k in packaged if k.startswith("batch_") and "@" not in k} <= set(best)
    assert log
