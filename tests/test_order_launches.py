"""The launches that etm_order_level is counted with (no GPU needed)."""

from __future__ import annotations

import pytest


@pytest.mark.parametrize("n,k,bits,want", [
    (0, 3, 12, 0), (1, 3, 12, 2), (2048, 9, 12, 2), (2049, 9, 12, 3), (65_536, 40, 12, 3),
    (65_537, 3, 12, 2 + 5 * 5),              # 36 bits of one word: five digits of a count, a scan of three and a scatter
    (65_537, 5, 12, 2 + 5 * 8),              # 60 bits
    (70_000_000, 6, 12, 2 + 1 + 5 * 8 + 1 + 5 * 2),  # two words, gathered first: 60 bits and 12
    (65_537, 2, 1, 2 + 5), (65_537, 65, 12, 0), (65_537, 3, 32, 0),
])
def test_launches_of_the_level_order(pkg, n, k, bits, want):
    assert pkg.load_library().etm_order_level_launches(n, k, bits) == want
