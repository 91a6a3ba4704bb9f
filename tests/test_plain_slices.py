"""How the FP64 sum cuts its atoms: slices of at least 512 atoms (all of them
where there are fewer), at most 4096 of them, and every SM's share of blocks
even."""
import math

import pytest

from mosaic_gb300.engine import plain_slices


@pytest.mark.parametrize("n", [1, 511, 513, 32_000, 8_000_000])
@pytest.mark.parametrize("bx", [1, 15, 742, 760, 761, 8192])
def test_slices(n, bx):
    s = plain_slices(n, bx, 152)
    assert 1 <= s <= max(1, min((n + 511) // 512, 4096))
    if n >= 1_000_000:                      # enough of them: under an eighth of the last wave empty
        blocks = bx * s / 152
        assert blocks / math.ceil(blocks) > 0.875
