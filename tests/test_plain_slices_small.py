"""How the FP64 sum cuts few atoms: the most laden SM of 152 never gets much
more than an even share of the blocks' time."""
import math

import pytest

from mosaic_gb300.engine import plain_slices


def _laden(n, bx, s):
    return math.ceil(bx * s / 152) * (n / s + 40.0)


@pytest.mark.parametrize("n", [513, 1_600, 2_500, 5_000, 20_000, 100_000])
@pytest.mark.parametrize("bx", [1, 8, 44, 77, 100, 153, 313])
def test_the_most_laden_sm_is_near_the_best(n, bx):
    s = plain_slices(n, bx, 152)
    most = (n + 511) // 512
    assert 1 <= s <= most
    best = min(_laden(n, bx, t) for t in range(1, most + 1))
    # one block an SM counts 1.2, and ten percent is not worth another cut; five
    # blocks an SM set up five times
    assert _laden(n, bx, s) <= 1.35 * best, (s, _laden(n, bx, s) / best)
