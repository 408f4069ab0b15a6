"""Mines whose small levels go through one launch: what the caller set, and what the general path gave, still holds."""

from __future__ import annotations

import gc
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


def _dense(pkg, n_items=120, n_rows=20_000, seed=5):
    import torch

    syn = pkg.synthetic
    p = np.minimum(syn.dense_k2_probs(n_items, seed=9) * 3, 0.9)
    bv = syn.bernoulli_bitvecs(syn.bernoulli_thresholds(p), n_rows, seed=seed)
    return torch.from_numpy(bv.view(np.int64)).cuda().view(torch.uint64), n_rows


def _launches(eng, *args, **kw):
    """The mine's output and the names of its timed launches."""
    eng.profile_kernels = True
    eng.reset_kernel_times()
    return eng.mine(*args, **kw), [e[0] for e in eng._events]


def _same_levels(a, b):
    assert len(a.levels) == len(b.levels) >= 2
    for x, y in zip(a.host_levels(), b.host_levels()):
        assert np.array_equal(x[0], y[0]) and np.array_equal(x[1], y[1])


@pytest.mark.parametrize("kw", [{}, {"tc_elem": 1}, {"tc_elem": 2}, {"tc_elem": 4 | 16}, {"pipeline": False},
                                {"deduction_bounds": False}])
def test_an_engine_set_up_to_count_otherwise_does(pkg, engm, kw):
    dev, n_rows = _dense(pkg)
    out, names = _launches(engm.Engine(**kw), dev, n_rows, 0.02, 4)
    assert ("mine_direct" in names) == (kw.get("tc_elem", 4) & ~16 == 4)
    ref = engm.Engine(method="popcount")
    _same_levels(out, ref.mine(dev, n_rows, 0.02, 4))


def test_a_launch_keeps_to_the_engines_budgets(pkg, engm, monkeypatch):
    """Levels of more candidates than a chunk go on in chunks; cut columns keep to the projection's bytes."""
    dev, n_rows = _dense(pkg)
    want, names = _launches(engm.Engine(), dev, n_rows, 0.02, 4)
    assert names == ["mine_direct"]
    most = max(s.n_candidates for s in want.stats[1:])
    eng = engm.Engine(chunk_cands=most // 4)
    got, names = _launches(eng, dev, n_rows, 0.02, 4)
    assert "level_compact" in names and eng.scratch.bufs["direct"].numel() * 4 < (2 << 20) + 6 * most
    _same_levels(got, want)
    for name in ("DIRECT_TURN", "DIRECT_PROJ_MIN", "DIRECT_LARGE"):
        monkeypatch.setattr(engm, name, 0)
    eng = engm.Engine(proj_bytes=1 << 12)
    _same_levels(eng.mine(dev, n_rows, 0.02, 4), want)
    n_items = len(want.gen_cols)
    assert eng.scratch.bufs["direct_proj"].numel() * 4 < (1 << 13) + 5 * (n_items + 64) * (n_items + 64)


def test_no_device_memory_for_a_launch_leaves_the_general_path(pkg, engm, monkeypatch):
    import torch

    dev, n_rows = _dense(pkg)
    want = engm.Engine().mine(dev, n_rows, 0.02, 4)
    eng = engm.Engine()
    get = eng.scratch.get

    def refuse(name, *args):
        if name.startswith("direct"):
            raise torch.OutOfMemoryError("no room")
        return get(name, *args)

    monkeypatch.setattr(eng.scratch, "get", refuse)
    got, names = _launches(eng, dev, n_rows, 0.02, 4)
    assert "mine_direct" not in names
    _same_levels(got, want)


@pytest.mark.parametrize("large", [False, True])
def test_a_limit_the_general_path_keeps_is_kept(pkg, engm, monkeypatch, large):
    """max_vram_gb a little above what the general path holds after any of its levels (the allocator rounds by up to a
    megabyte a buffer)."""
    import torch

    gc.collect()
    dev, n_rows = _dense(pkg)
    if large:
        monkeypatch.setattr(engm, "DIRECT_LARGE", 0)
    seen = []
    monkeypatch.setattr(engm, "check_memory_guard", lambda k, ram, vram, *limits: seen.append(vram))
    general = engm.Engine()
    general.direct = False
    want = general.mine(dev, n_rows, 0.02, 4, max_vram_gb=1e9)
    used = max(seen) - engm._allocated_gb(dev.device)
    monkeypatch.undo()
    if large:
        monkeypatch.setattr(engm, "DIRECT_LARGE", 0)
    del general
    held = sum(t.numel() * t.element_size() for lv in want.levels for t in (lv.rows, lv.counts)) / 2**30
    limit = engm._allocated_gb(dev.device) + used + held + 6 / 1024
    got = engm.Engine().mine(dev, n_rows, 0.02, 4, max_vram_gb=limit)
    _same_levels(got, want)
    torch.cuda.synchronize()


@pytest.mark.parametrize("support,few", [(0.05, True), (0.02, False)])
def test_a_result_holds_little_more_than_its_bytes(pkg, engm, support, few):
    gc.collect()
    dev, n_rows = _dense(pkg)
    eng = engm.Engine()
    eng.mine(dev, n_rows, support, 4)
    before = engm._allocated_gb(dev.device)
    kept = [eng.mine(dev, n_rows, support, 4) for _ in range(8)]
    own = sum(t.numel() * t.element_size() for out in kept for lv in out.levels for t in (lv.rows, lv.counts))
    assert all((out.host is not None) == few for out in kept)
    assert (engm._allocated_gb(dev.device) - before) * 2**30 < own + 8 * (4 * (engm.DIRECT_FETCH_COUNTS + engm.DIRECT_FETCH_ROWS) + 1024)


def test_a_servers_requests_keep_their_launches_to_the_budget(pkg, engm, monkeypatch):
    """A slot's footprint holds its direct launches' buffers; a tight budget gets small ones."""
    serve = import_module(pkg.__name__ + ".serve")
    monkeypatch.setattr(engm, "DIRECT_LARGE", 0)
    dev, n_rows = _dense(pkg)
    counts = np.array([int(x) for x in engm.Engine().column_counts(dev.data_ptr(), dev.shape[0], dev.shape[1], dev.shape[1])])
    ds = serve.Dataset(dev, np.arange(dev.shape[0]), n_rows, counts)
    engines = []

    class Kept(engm.Engine):
        def __init__(self, **kw):
            super().__init__(**kw)
            engines.append(self)

    monkeypatch.setattr(serve, "Engine", Kept)
    want = engm.Engine().mine(dev, n_rows, 0.02, 4).host_levels()
    large = engm.direct_need(len(counts), len(counts), int(dev.shape[1]), 1 << 24, 1 << 30)
    assert large > 200 << 20
    for budget in (8 << 30, 256 << 20):
        engines.clear()
        with serve.Server([ds], slots=2, hbm_budget=budget) as server:
            need = server.footprint(0, 0.02)
            got = server.submit(0, 0.02, 4).result(timeout=120).levels
        held = max(e._direct_held() for e in engines)
        assert held <= need <= max(budget // 2, 160 << 20)
        assert (held > 200 << 20) == (budget == 8 << 30)
        for (a, n), (b, m) in zip(got, want):
            assert np.array_equal(a, b) and np.array_equal(n, m)


@pytest.mark.parametrize("by_support", [False, True])
def test_the_memory_guards_read_level_by_level(pkg, engm, monkeypatch, by_support):
    """Each level of a launch is checked with what the mine holds up to it, and the limit is named after the level that
    passes it."""
    gc.collect()
    dev, n_rows = _dense(pkg)
    if by_support:
        monkeypatch.setattr(engm, "DIRECT_TURN", 0)
    eng = engm.Engine()
    want = eng.mine(dev, n_rows, 0.02, 4)
    check, seen = engm.check_memory_guard, []
    monkeypatch.setattr(engm, "check_memory_guard", lambda k, ram, vram, *limits: seen.append((k, vram)))
    eng.mine(dev, n_rows, 0.02, 4, max_vram_gb=1e9)
    assert [k for k, _ in seen] == [2, 3, 4]
    sizes = {lv.k: 4 * lv.n * (lv.k + 1) / 2**30 * (2 if by_support else 1) for lv in want.levels}
    for (_, a), (k, b) in zip(seen, seen[1:]):
        if k > 3 or not by_support:
            assert abs(b - a - sizes[k]) < 1e-9
    monkeypatch.setattr(engm, "check_memory_guard", check)
    eng._drop_direct = lambda: 0.0
    for k in () if by_support else (3, 4):  # the other leaves its order before it gives up
        limit = (dict(seen)[k - 1] + dict(seen)[k]) / 2
        with pytest.raises(MemoryError, match=f"after K={k}"):
            eng.mine(dev, n_rows, 0.02, 4, max_vram_gb=limit)


def test_a_large_result_stays_on_the_device(pkg, engm, monkeypatch):
    """One launch's result past what comes back with its header: level 1 alone is copied, the frame is made on the device."""
    monkeypatch.setattr(engm, "DIRECT_FETCH_COUNTS", 512)
    monkeypatch.setattr(engm, "DIRECT_FETCH_ROWS", 1024)
    dev, n_rows = _dense(pkg)
    items = np.arange(dev.shape[0], dtype=np.int64) * 3 + 1
    for support, small in ((0.1, True), (0.02, False)):
        out, names = _launches(engm.Engine(), dev, n_rows, support, 4)
        assert names == ["mine_direct"] and (out.host is not None) == small
        general = engm.Engine()
        general.direct = False
        want = general.mine(dev, n_rows, support, 4)
        _same_levels(out, want)
        for a, b in zip(out.frame_arrays(items)[:3], want.frame_arrays(items)[:3]):
            assert np.array_equal(a, b)
    monkeypatch.setattr(engm, "DIRECT_FETCH_COUNTS", 8)  # fewer than the columns
    out = engm.Engine().mine(dev, n_rows, 0.02, 4)
    assert out.host is None and np.array_equal(out.level1_counts, want.level1_counts)
    _same_levels(out, want)


@pytest.mark.parametrize("kw", [{"prune_equal_support": True}, {"use_generator_pruning": True}, {}])
@pytest.mark.parametrize("path", ["launch", "turn", "ordered", "resume"])
def test_returned_levels_carry_their_free_flags(pkg, engm, monkeypatch, path, kw):
    """As the general path returns them: from a launch, in another order than the columns', and of a resumed mine."""
    import torch

    dev, n_rows = _dense(pkg)
    bits = dev.view(torch.int64)
    bits[50], bits[70], bits[90] = bits[3] & bits[5], bits[7], bits[2] | bits[11]  # sets with supersets of their count
    general = engm.Engine()
    general.direct = general.by_support = False
    want = general.mine(dev, n_rows, 0.02, 5, **kw)
    if path == "turn":
        monkeypatch.setattr(engm, "DIRECT_TURN", 0)
    elif path == "ordered":
        monkeypatch.setattr(engm, "ORDER_WORDS", 0)
        monkeypatch.setattr(engm, "DIRECT_WORDS", 1 << 22)
    resume = None
    if path == "resume":
        level = want.levels[0]
        resume = (2, want.gen_cols[level.rows.cpu().numpy()], level.counts.cpu().numpy())
    got = engm.Engine().mine(dev, n_rows, 0.02, 5, resume=resume, **kw)
    levels = want.levels[1:] if path == "resume" else want.levels
    assert len(got.levels) == len(levels) >= 2
    for a, b in zip(got.levels, levels):
        assert torch.equal(a.rows, b.rows) and torch.equal(a.counts, b.counts)
        assert (a.free is None) == (b.free is None) == (not kw)
        if kw:
            assert torch.equal(a.free, b.free)
    if "use_generator_pruning" in kw:
        assert any((lv.free == 0).any() for lv in levels)
    got = engm.Engine().mine(dev, n_rows, 0.02, 5, resume=resume, free_flags=False, **kw)
    assert all(torch.equal(a.rows, b.rows) for a, b in zip(got.levels, levels))


@pytest.mark.parametrize("kw", [{"tc_elem": 1}, {"tc_elem": 2}, {"pipeline": False}, {"deduction_bounds": False}])
def test_counting_by_support_asks_for_no_operands(pkg, engm, monkeypatch, kw):
    """The generators' order while counting is the same in any format of the operands, pipelined or not."""
    monkeypatch.setattr(engm, "ORDER_WORDS", 0)
    monkeypatch.setattr(engm, "DIRECT_WORDS", 0)
    dev, n_rows = _dense(pkg)
    out, names = _launches(engm.Engine(**kw), dev, n_rows, 0.02, 4)
    assert "order_level" in names and "gram_tc" in names
    _same_levels(out, engm.Engine(method="popcount").mine(dev, n_rows, 0.02, 4))


def test_buffers_of_a_mine_with_more_room_are_given_back(pkg, engm, monkeypatch):
    monkeypatch.setattr(engm, "DIRECT_LARGE", 0)
    dev, n_rows = _dense(pkg)
    eng = engm.Engine()
    want = eng.mine(dev, n_rows, 0.02, 4)
    assert eng._direct_held() > 100 << 20
    for room in (48 << 20, 1 << 20):
        eng.direct_max_bytes = room
        _same_levels(eng.mine(dev, n_rows, 0.02, 4), want)
        assert eng._direct_held() <= room
