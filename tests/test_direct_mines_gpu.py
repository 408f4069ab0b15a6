"""Mines whose small levels go through one launch: what the caller set, and what the general path gave, still holds."""

from __future__ import annotations

from importlib import import_module
from itertools import combinations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def engm(pkg):
    return import_module(pkg.__name__ + ".engine")


def _ones(n_items, n_rows):
    """Columns that hold every row."""
    import torch

    bits = np.zeros((n_items, -(-n_rows // 64) * 64), np.uint8)
    bits[:, :n_rows] = 1
    bv = np.packbits(bits, axis=1, bitorder="little").view(np.int64)
    return torch.from_numpy(bv).cuda().view(torch.uint64)


def test_levels_past_the_launchs_longest_itemset(engm):
    """A level of 61 items resumed: the launch's own limit is 62 items, the mine's 63."""
    n_items, n_rows, k = 64, 100, 61
    drop = np.array(list(combinations(range(n_items), n_items - k)))
    rows = np.array([np.setdiff1d(np.arange(n_items), d) for d in drop])
    out = engm.Engine().mine(_ones(n_items, n_rows), n_rows, 0.5, 63, resume=(k, rows, np.full(len(rows), n_rows)))
    assert [(lv.k, lv.n) for lv in out.levels] == [(62, 2016), (63, 64)]
    assert all((lv.counts == n_rows).all() for lv in out.levels)
