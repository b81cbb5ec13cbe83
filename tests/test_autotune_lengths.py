"""The autotuner's lengths for the tile kernel are lengths that run it."""
import math

import pytest

from jtransforms_gb300 import autotune


@pytest.mark.parametrize("lg", range(4, 14))
def test_tile_lengths_run_the_tile_kernel(lg):
    for n in autotune.tile_lengths(lg):
        assert math.ceil(math.log2(n)) == lg
        m = n
        for p in (2, 3, 5, 7, 11, 13):
            while m % p == 0:
                m //= p
        # register passes take 2..13 (float) and 2..7 (double); floats of one pass (up to 16) keep the tile form
        assert m > 1 or n <= 16
        assert m <= 61
