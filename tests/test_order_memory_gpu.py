"""Mines that count over generators in ascending support hold their levels in two orders: under a limit of device memory that
the columns' order keeps, and with no room to sort a level whole. Against the columns' order; zero tolerance."""

from __future__ import annotations

import gc
from importlib import import_module

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MODES = [{}, {"prune_equal_support": True}, {"use_generator_pruning": True}]


@pytest.fixture
def engm(pkg):
    return import_module(pkg.__name__ + ".engine")


def _table(pkg, n_items=300):
    import torch

    syn = pkg.synthetic
    p = np.minimum(syn.dense_k2_probs(n_items, seed=2) * 2.5, 0.9)
    bv = syn.bernoulli_bitvecs(syn.bernoulli_thresholds(p), 30_011, seed=3)
    bv[7] = bv[8]
    return torch.from_numpy(bv.view(np.int64)).cuda().view(torch.uint64), 30_011


def _same(a, b):
    import torch

    assert len(a.levels) == len(b.levels) >= 3
    for x, y in zip(a.levels, b.levels):
        assert torch.equal(x.rows, y.rows) and torch.equal(x.counts, y.counts)
    assert [(t.k, t.n_candidates, t.n_frequent, t.n_groups) for t in a.stats] == \
        [(t.k, t.n_candidates, t.n_frequent, t.n_groups) for t in b.stats]


def _guarded(engm, monkeypatch, eng, *args, **kw):
    """The mine and its readings of device memory by level, from where it began, without the direct launches' buffers."""
    import torch

    seen = []
    eng._drop_direct()
    before = engm._allocated_gb(torch.device("cuda"))
    with monkeypatch.context() as m:
        m.setattr(engm, "check_memory_guard", lambda k, ram, vram, *limits: seen.append(vram - before - eng._direct_held() / 2**30))
        out = eng.mine(*args, max_vram_gb=1e9, **kw)
    eng._drop_direct()
    return out, seen


@pytest.mark.parametrize("kw", MODES)
@pytest.mark.parametrize("direct", [0, 1 << 23])
@pytest.mark.parametrize("keep", [True, False])
def test_a_limit_the_columns_order_keeps_is_kept(pkg, engm, monkeypatch, direct, keep, kw):
    """The mine leaves the other order when it passes the limit, after a level or between the levels of one launch."""
    gc.collect()
    dev, n_rows = _table(pkg)
    monkeypatch.setattr(engm, "ORDER_WORDS", 0)
    monkeypatch.setattr(engm, "DIRECT_WORDS", direct)
    monkeypatch.setattr(engm, "DIRECT_TURN", 0)
    plain, ordered = engm.Engine(), engm.Engine()
    plain.by_support = False
    for eng in (plain, ordered):  # their scratch is there
        eng.mine(dev, n_rows, 0.006, 4, **kw)
    want = plain.mine(dev, n_rows, 0.006, 4, **kw)
    _same(ordered.mine(dev, n_rows, 0.006, 4, **kw), want)
    want_on = [(lv.k, lv.rows.cpu().numpy(), lv.counts.cpu().numpy()) for lv in want.levels]
    levels = []
    on = {} if keep else dict(on_level=lambda *level: levels.append(level), keep_levels=False)
    _, low = _guarded(engm, monkeypatch, plain, dev, n_rows, 0.006, 4, **on, **kw)
    _, high = _guarded(engm, monkeypatch, ordered, dev, n_rows, 0.006, 4, **on, **kw)
    assert max(high) > max(low) + 0.01  # GB: the allocator rounds by a megabyte a buffer
    levels.clear()
    left = []
    gather = engm.Engine.gather
    monkeypatch.setattr(engm.Engine, "gather", lambda self, *a: (left.append(len(a)), gather(self, *a))[1])
    limit = engm._allocated_gb(dev.device) + (max(low) + max(high)) / 2
    got = ordered.mine(dev, n_rows, 0.006, 4, max_vram_gb=limit, **on, **kw)
    assert len(left) == 2  # the generating columns gathered again
    if keep:
        _same(got, want)
    else:
        assert len(levels) == len(want_on) + 1
        for (k, rows, counts), (k2, r2, c2) in zip(levels[1:], want_on):
            assert k == k2 and np.array_equal(rows, want.gen_cols[r2]) and np.array_equal(counts, c2)


@pytest.mark.parametrize("kw", MODES)
@pytest.mark.parametrize("rows,piece,step", [(1000, 40_000, 77_777), (1000, 1 << 27, 1 << 24), (None, 50_000, 40_960)])
def test_a_level_sorted_in_pieces(pkg, engm, monkeypatch, rows, piece, step, kw):
    """Levels of more rows than are sorted at once, and levels that leave no room for it (rows None)."""
    import torch

    dev, n_rows = _table(pkg)
    plain, ordered = engm.Engine(), engm.Engine()
    plain.by_support = False
    want = plain.mine(dev, n_rows, 0.006, 4, **kw)
    monkeypatch.setattr(engm, "ORDER_WORDS", 0)
    monkeypatch.setattr(engm, "DIRECT_WORDS", 0)
    monkeypatch.setattr(engm, "ORDER_PIECE", piece)
    monkeypatch.setattr(engm, "ORDER_STEP", step)
    most = []
    if rows is not None:
        monkeypatch.setattr(engm, "ORDER_ROWS", rows)
    sort = engm.Engine._order_rows

    def limited(self, level_rows, *args):
        if rows is None and len(level_rows) > 600_000:
            raise torch.OutOfMemoryError("no room")
        most.append(len(level_rows))
        sort(self, level_rows, *args)

    monkeypatch.setattr(engm.Engine, "_order_rows", limited)
    _same(ordered.mine(dev, n_rows, 0.006, 4, **kw), want)
    assert len(most) > 6 or piece > 50_000


@pytest.mark.parametrize("kw", MODES)
@pytest.mark.parametrize("keep", [True, False])
def test_the_limit_is_passed_within_a_launch(pkg, engm, monkeypatch, keep, kw):
    """The levels past 2 come out of one launch over generators in ascending support, which takes both orders' memory."""
    import torch

    gc.collect()
    dev, n_rows = _table(pkg, 200)
    monkeypatch.setattr(engm, "DIRECT_LARGE", 0)
    monkeypatch.setattr(engm, "DIRECT_TURN", 0)
    monkeypatch.setattr(engm, "DIRECT_WORDS", 1 << 36)
    # What is held without the allocator's rounding, and room for the launch itself.
    monkeypatch.setattr(engm, "_allocated_gb", lambda device: torch.cuda.memory_stats(device)[
        "requested_bytes.all.current"] / 2**30)
    monkeypatch.setattr(engm.Engine, "_direct_room", lambda self, limit: float("inf"))
    plain, ordered = engm.Engine(), engm.Engine()
    plain.direct = plain.by_support = False
    want = plain.mine(dev, n_rows, 0.006, 4, **kw)
    ordered.profile_kernels = True
    _same(ordered.mine(dev, n_rows, 0.006, 4, **kw), want)
    assert [e[0] for e in ordered._events if e[0] in ("mine_direct", "gram_tc")] == ["mine_direct", "mine_direct"]
    ordered.profile_kernels = False
    want_on = [(lv.k, want.gen_cols[lv.rows.cpu().numpy()], lv.counts.cpu().numpy()) for lv in want.levels]
    levels = []
    on = {} if keep else dict(on_level=lambda *level: levels.append(level), keep_levels=False)
    _, high = _guarded(engm, monkeypatch, ordered, dev, n_rows, 0.006, 4, **on, **kw)
    levels.clear()
    left = []
    gather = engm.Engine.gather
    monkeypatch.setattr(engm.Engine, "gather", lambda self, *a: (left.append(len(a)), gather(self, *a))[1])
    # Every level of the launch once, and those up to 3 twice: past that the other order is left.
    once = [4 * lv.n * (lv.k + 1) / 2**30 for lv in want.levels]
    assert high[-1] - high[0] > 1.5 * sum(once[1:]) and min(once[1:]) > 0.003 and len(once) == 3
    limit = engm._allocated_gb(dev.device) + high[1] + sum(once[2:]) + 0.003
    assert limit - engm._allocated_gb(dev.device) < high[-1] - 0.003
    got = ordered.mine(dev, n_rows, 0.006, 4, max_vram_gb=limit, **on, **kw)
    assert len(left) == 2
    if keep:
        _same(got, want)
    else:
        assert len(levels) == len(want_on) + 1
        for (k, rows, counts), (k2, r2, c2) in zip(levels[1:], want_on):
            assert k == k2 and np.array_equal(rows, r2) and np.array_equal(counts, c2)
