"""Levels mined by one cooperative launch (etm_mine_direct) against the general path and the oracle, at the sizes where
it can go wrong: word tails and slabs, tiles of 8, 16- and 8-byte columns, levels handed over at its limits, and the tail of a mine."""

from __future__ import annotations

from importlib import import_module

import numpy as np
import pytest

from oracle import miner

pytestmark = pytest.mark.gpu


def _mine(eng, bv, n_rows, s, k, **kw):
    import torch

    dev = torch.from_numpy(np.ascontiguousarray(bv).view(np.int64)).cuda().view(torch.uint64)
    return eng.mine(dev, n_rows, s, k, **kw)


def _same(a, b):
    la, lb = a.host_levels(), b.host_levels()
    assert len(la) == len(lb)
    for (ra, ca), (rb, cb) in zip(la, lb):
        assert np.array_equal(ra, rb) and np.array_equal(ca, cb)
    assert [(s.k, s.n_candidates, s.n_frequent) for s in a.stats] == [(s.k, s.n_candidates, s.n_frequent) for s in b.stats]


MODES = [{}, {"prune_equal_support": True}, {"use_generator_pruning": True}]


@pytest.mark.parametrize("kw", MODES)
@pytest.mark.parametrize("n_rows,n_items", [(1, 3), (63, 5), (64, 17), (65, 18), (2049, 33), (8191, 24), (8193, 25),
                                            (40_001, 12), (65_536, 10)])
def test_whole_mines_match_the_general_path_and_the_oracle(pkg, n_rows, n_items, kw):
    engm = import_module(pkg.__name__ + ".engine")
    rng = np.random.default_rng(n_rows)
    p = rng.uniform(0.05, 0.7, n_items)
    bits = rng.random((n_items, n_rows)) < p[:, None]
    bits[0] = True  # an item in every row
    if n_items > 4:
        bits[3] = bits[4]  # equal supports
    words = -(-n_rows // 64)
    padded = np.zeros((n_items, words * 64), bool)
    padded[:, :n_rows] = bits
    bv = np.packbits(padded.reshape(n_items, words, 64), axis=2, bitorder="little").view(np.uint64)[:, :, 0].copy()
    general = engm.Engine()
    general.direct = False
    small = engm.Engine()
    out = _mine(small, bv, n_rows, 0.08, 7, **kw)
    assert out.host is not None  # one launch
    _same(out, _mine(general, bv, n_rows, 0.08, 7, **kw))
    ref = miner.mine_bitvecs(bv, n_rows, 0.08, 7, **kw)
    want = miner.canonical(ref.levels, np.arange(n_items))
    levels = out.host_levels()
    have = sorted(((tuple(int(x) for x in r), int(c)) for rows, counts in levels for r, c in zip(rows, counts)),
                  key=lambda t: (len(t[0]), t[0]))
    assert have == want


@pytest.mark.parametrize("kw", MODES)
@pytest.mark.parametrize("limit", [0, 60_000, 400_000])
def test_levels_past_the_limit_go_on_on_the_general_path(pkg, monkeypatch, limit, kw):
    """A work limit that stops the launch before K=2, or before a later level; the mine's tail is small again."""
    engm = import_module(pkg.__name__ + ".engine")
    syn = pkg.synthetic
    t = syn.plain_small(n_rows=20_000, n_items=300, seed=5)
    uniq, inv = np.unique(t.items, return_inverse=True)
    bv = miner.bitvecs_from_csr(t.indptr, inv.astype(np.int32), len(uniq), t.n_rows)
    general = engm.Engine()
    general.direct = False
    want = _mine(general, bv, t.n_rows, 0.004, None, **kw)
    monkeypatch.setattr(engm, "DIRECT_WORDS", limit)
    got = _mine(engm.Engine(), bv, t.n_rows, 0.004, None, **kw)
    assert got.host is None and len(got.levels) >= 3
    _same(got, want)


def test_small_outputs_and_too_many_columns_fall_back(pkg, monkeypatch):
    """More frequent columns than a direct level holds, and a level that does not fit the outputs."""
    engm = import_module(pkg.__name__ + ".engine")
    rng = np.random.default_rng(3)
    n_rows, n_items = 640, engm.DIRECT_ROWS + 40
    bv = np.zeros((n_items, 10), np.uint64)
    bv[:, rng.integers(0, 10, 4)] = np.uint64(2**64 - 1)
    bv[20:] = 0
    bv[np.arange(20, n_items), rng.integers(0, 10, n_items - 20)] = np.uint64(1)
    general = engm.Engine()
    general.direct = False
    _same(_mine(engm.Engine(), bv, n_rows, 1 / 640, 2), _mine(general, bv, n_rows, 1 / 640, 2))
    p = rng.uniform(0.3, 0.7, 60)
    wide = np.packbits((rng.random((60, 10, 64)) < p[:, None, None]), axis=2, bitorder="little").view(np.uint64)[:, :, 0]
    want = _mine(general, wide, n_rows, 0.05, 4)
    monkeypatch.setattr(engm, "DIRECT_COUNTS_CAP", engm.DIRECT_ROWS + 5)
    got = _mine(engm.Engine(), wide, n_rows, 0.05, 4)
    assert got.host is None
    _same(got, want)


@pytest.mark.parametrize("kw", MODES)
@pytest.mark.parametrize("n_rows,lo,hi,s,k", [(262_143, 0.03, 0.1, 2e-5, 4), (262_145, 0.001, 0.003, 1 / 262_145, 5),
                                              (245_760, 0.01, 0.4, 4e-4, 4), (278_600, 0.02, 0.09, 1e-4, 5)])
def test_levels_over_columns_cut_to_the_first_item(pkg, monkeypatch, n_rows, lo, hi, s, k, kw):
    """K>=3 on projected columns: whole and ragged segments, first items of a few rows a segment and of most of it, and a
    level past the offsets in shared memory; from a level 2 turned to ascending support."""
    engm = import_module(pkg.__name__ + ".engine")
    rng = np.random.default_rng(n_rows)
    n_items, words = 54, -(-n_rows // 64)
    assert n_items * (n_items - 1) * (n_items - 2) // 6 * words >= 1 << 26  # all pairs frequent: the level is projected
    p = rng.uniform(lo, hi, n_items)
    p[7], p[31] = 0.6, 0.2
    bits = rng.random((n_items, words * 64), dtype=np.float32) < p[:, None]
    bits[:, n_rows:] = False
    bits[20] = bits[21]  # equal supports
    bv = np.packbits(bits.reshape(n_items, words, 64), axis=2, bitorder="little").view(np.uint64)[:, :, 0].copy()
    general = engm.Engine()
    general.direct = False
    general.by_support = False
    want = _mine(general, bv, n_rows, s, k, **kw)
    monkeypatch.setattr(engm, "DIRECT_TURN", 0)
    monkeypatch.setattr(engm, "DIRECT_PROJ_MIN", 0)
    monkeypatch.setattr(engm, "DIRECT_LARGE", 0)
    eng = engm.Engine()
    _same(_mine(eng, bv, n_rows, s, k, **kw), want)
    for rows in (512, 4096):  # levels past a launch's memory go on in a larger one, on the same projected columns
        monkeypatch.setattr(engm, "DIRECT_ROWS", rows)
        _same(_mine(eng, bv, n_rows, s, k, **kw), want)
    monkeypatch.setattr(engm, "DIRECT_WORDS", 200_000)  # K=2 past it, and a projected level
    _same(_mine(eng, bv, n_rows, s, k, **kw), want)


@pytest.mark.parametrize("room_gb", [0.09, 0.4])
def test_a_tight_memory_limit_takes_small_launches(pkg, room_gb):
    """A limit of device memory that a large launch's buffers would pass: the mine goes on in small ones (at first with
    nothing but these, then with some of the large ones) and the limit is kept."""
    import torch

    engm = import_module(pkg.__name__ + ".engine")
    rng = np.random.default_rng(9)
    n_rows, n_items = 262_080, 600  # 2.5 M words: a large launch by its input
    p = np.concatenate([rng.uniform(0.04, 0.09, 54), np.full(n_items - 54, 1e-4)])
    bits = np.zeros((n_items, n_rows), np.uint8)
    for c in range(n_items):
        bits[c, rng.random(n_rows, dtype=np.float32) < p[c]] = 1
    bv = np.packbits(bits, axis=1, bitorder="little").view(np.uint64)
    general = engm.Engine()
    general.direct = general.by_support = False
    want = _mine(general, bv, n_rows, 1e-3, 4)
    del general
    torch.cuda.empty_cache()
    dev = torch.from_numpy(bv.view(np.int64)).cuda().view(torch.uint64)
    limit = engm._allocated_gb(dev.device) + room_gb
    got = engm.Engine().mine(dev, n_rows, 1e-3, 4, max_vram_gb=limit)
    _same(got, want)


def test_medium_results_reuse_two_page_locked_buffers(pkg, monkeypatch):
    """Results between the medium and the large size: at most two buffers, never that of a live result, of any order of
    sizes and drops."""
    engm = import_module(pkg.__name__ + ".engine")
    pool = engm._PinnedPool()
    import torch

    monkeypatch.setattr(engm, "_PINNED", pool)
    monkeypatch.setattr(engm, "PINNED_MEDIUM_BYTES", 0)
    live = {}
    rng = np.random.default_rng(0)
    for step in range(40):
        n = int(rng.integers(1, 5000))
        t = torch.arange(n, dtype=torch.int64, device="cuda") + step
        live[step % 5] = (step, engm._copy_to_host(t, t.to(torch.float64)))
        if rng.random() < 0.4:
            live.pop(int(rng.integers(0, 5)), None)
        assert len(pool.medium) <= engm.PINNED_MEDIUM_BUFFERS and not pool.entries
        for at, (a, b) in live.values():
            assert a[0] == at and np.array_equal(a, np.arange(len(a)) + at) and np.array_equal(a, b)
