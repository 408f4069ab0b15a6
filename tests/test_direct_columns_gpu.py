"""Levels counted on columns cut to the first item (project_columns of etm_mine_direct), on tables whose rows are not dealt at
random: items that live in some segments of the rows and not in others. Against the general path; zero tolerance."""

from __future__ import annotations

from importlib import import_module

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SEG_ROWS = 256 * 64  # rows of a projection segment
N_ITEMS = 54


def _bitvecs(bits, words):
    return np.packbits(bits.reshape(len(bits), words, 64), axis=2, bitorder="little").view(np.uint64)[:, :, 0].copy()


def _runs(rng, n_rows, rows_a_segment, live, last_empty):
    """Items over ``live`` of the segments each, with about ``rows_a_segment`` rows in one of those."""
    words = -(-n_rows // 64)
    n_seg = -(-words // 256)
    bits = rng.random((N_ITEMS, words * 64), dtype=np.float32) < rows_a_segment / SEG_ROWS
    for i in range(N_ITEMS):
        off = rng.permutation(n_seg)[: n_seg - max(1, round(live * n_seg))]
        for s in off:
            bits[i, s * SEG_ROWS:(s + 1) * SEG_ROWS] = False
    if last_empty:
        bits[:, (n_seg - 1) * SEG_ROWS:] = False
    bits[:, n_rows:] = False
    return bits, words


def _projected(bits, words, mc):
    """Whether etm_mine_direct cuts these columns: its two conditions, from the pairs that are frequent."""
    order = np.argsort(bits.sum(1), kind="stable")
    x = bits[order].astype(np.float32)
    pairs = np.triu((x @ x.T) >= mc, 1)
    m = pairs.sum(1)
    per_seg = np.add.reduceat(bits[order], np.arange(0, bits.shape[1], SEG_ROWS), axis=1)
    cut = (-(-per_seg // 128) * 2).sum(1)  # words of an item's rows, each segment's filled up to 16 bytes
    return (int((m * (m - 1) // 2).sum()) * words >= 1 << 26 and
            int((m * cut)[m > 1].sum()) * 8 <= int(m.sum()) * words)


def _check(pkg, monkeypatch, bits, words, n_rows, mc, k):
    import torch

    engm = import_module(pkg.__name__ + ".engine")
    assert _projected(bits, words, mc)
    dev = torch.from_numpy(_bitvecs(bits, words).view(np.int64)).cuda().view(torch.uint64)
    general = engm.Engine()
    general.direct = general.by_support = False
    want = general.mine(dev, n_rows, mc / n_rows, k)
    assert len(want.levels) >= 2
    for name in ("DIRECT_TURN", "DIRECT_PROJ_MIN", "DIRECT_LARGE"):
        monkeypatch.setattr(engm, name, 0)
    eng = engm.Engine()
    for _ in range(3):  # again on the memory that the launch before left
        got = eng.mine(dev, n_rows, mc / n_rows, k)
        assert len(got.levels) == len(want.levels)
        for a, b in zip(got.levels, want.levels):
            assert torch.equal(a.rows, b.rows) and torch.equal(a.counts, b.counts)


@pytest.mark.parametrize("n_rows,rows_a_segment,live,last_empty", [
    (18 * SEG_ROWS, 700, 0.6, True),         # segments without a row, in the middle and at the end
    (17 * SEG_ROWS + 1, 700, 1.0, False),    # a last segment of one row, which most items do not hold
    (24 * SEG_ROWS - 61, 1500, 0.3, True),   # most segments empty, the list of rows flushed within a segment
    (17 * SEG_ROWS + 64 * 3, 900, 0.6, False),
])
def test_segments_without_a_row(pkg, monkeypatch, n_rows, rows_a_segment, live, last_empty):
    rng = np.random.default_rng(n_rows + rows_a_segment)
    bits, words = _runs(rng, n_rows, rows_a_segment, live, last_empty)
    _check(pkg, monkeypatch, bits, words, n_rows, 4, 5)


@pytest.mark.parametrize("rows_a_segment", [1, 3, 8, 60, 130])
def test_first_items_of_few_rows_a_segment(pkg, monkeypatch, rows_a_segment):
    """Items that share their rows, from one row of 16,384 on: pairs are frequent although the items are rare."""
    rng = np.random.default_rng(rows_a_segment)
    n_rows = 40 * SEG_ROWS - 100
    words = -(-n_rows // 64)
    pool = rng.random(words * 64) < 1.25 * rows_a_segment / SEG_ROWS
    bits = (rng.random((N_ITEMS, words * 64), dtype=np.float32) < 0.8) & pool
    bits[:, n_rows:] = False
    _check(pkg, monkeypatch, bits, words, n_rows, max(2, int(0.5 * bits[0].sum())), 3)
