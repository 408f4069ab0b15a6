"""Mines counted over generators in ascending support: the levels come back in the columns' order, rows, counts, stats
and callbacks alike. etm_order_level and etm_group_totals against numpy. Zero tolerance."""

from __future__ import annotations

import ctypes
from importlib import import_module

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _level(rng, n, k, n_items):
    """n distinct ascending k-itemsets over n_items, in random order, one per row."""
    rows = np.sort(np.argpartition(rng.random((2 * n + 8, n_items)), k - 1, axis=1)[:, :k], axis=1) if k > 2 else None
    if k <= 2:
        rows = np.sort(rng.integers(0, n_items, (4 * n + 64, k)), axis=1)
        rows = rows[rows[:, 0] < rows[:, -1]] if k == 2 else rows
    rows = np.unique(rows, axis=0)
    return rng.permutation(rows)[:n].astype(np.int32)


@pytest.mark.parametrize("n,k,n_items", [(1, 1, 1), (1, 3, 5), (2, 2, 4), (33, 1, 900), (257, 3, 40), (4000, 9, 60),
                                         (3000, 17, 40), (16_384, 2, 5000), (16_385, 2, 5000), (16_385, 4, 70_000),
                                         (24_577, 3, 4096), (2048, 5, 40), (2049, 5, 40), (2049, 2, 300), (65_536, 8, 24), (65_537, 8, 24), (12_000, 8, 16), (70_001, 6, 30), (40_000, 11, 300), (20_000, 23, 50)])
def test_level_order_matches_numpy(pkg, n, k, n_items):
    import torch

    lib = pkg.load_library()
    rng = np.random.default_rng(n + k)
    if n * n_items > 1 << 28:  # wide rows: ascending draws instead of partitions
        rows = np.unique(np.sort(rng.integers(0, n_items, (n + 50, k)), axis=1), axis=0)
        rows = rng.permutation(rows[(np.diff(rows, axis=1) > 0).all(axis=1)])[:n].astype(np.int32)
    else:
        rows = _level(rng, n, k, n_items)
    n = len(rows)
    counts = rng.integers(0, 2**31 - 1, n).astype(np.int32)
    perm = rng.permutation(n_items).astype(np.int32)
    want = np.sort(perm[rows], axis=1)
    at = np.lexsort(want.T[::-1])
    bits = max(1, (n_items - 1).bit_length())
    need = ctypes.c_int64()
    assert lib.etm_order_level_bytes(n, k, bits, ctypes.byref(need)) == 0
    d = [torch.from_numpy(x).cuda() for x in (rows, counts, perm)]
    out_r, out_c = torch.empty_like(d[0]), torch.empty_like(d[1])
    scratch = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    args = (d[0].data_ptr(), d[1].data_ptr(), n, k, d[2].data_ptr(), bits, out_r.data_ptr(), out_c.data_ptr(),
            scratch.data_ptr())
    assert lib.etm_order_level(*args, need.value - 1, stream) == 3
    assert lib.etm_order_level(*args, need.value, stream) == 0, lib.etm_last_error()
    assert np.array_equal(out_r.cpu().numpy(), want[at])
    assert np.array_equal(out_c.cpu().numpy(), counts[at])
    # The groups of the ordered level.
    tot = torch.empty(2, dtype=torch.int64, device="cuda")
    assert lib.etm_group_totals(out_r.data_ptr(), n, k, tot.data_ptr(), stream) == 0, lib.etm_last_error()
    if k == 1:
        sizes = np.array([n])
    else:
        _, sizes = np.unique(want[:, :-1], axis=0, return_counts=True)
    assert tot.cpu().tolist() == [int((sizes * (sizes - 1) // 2).sum()), int((sizes >= 2).sum())]


@pytest.mark.parametrize("kw", [{}, {"prune_equal_support": True}, {"use_generator_pruning": True}])
@pytest.mark.parametrize("direct_words", [0, 200_000])
@pytest.mark.parametrize("data", ["dense", "zipf"])
def test_mines_match_the_columns_order(pkg, monkeypatch, data, direct_words, kw):
    """Against an engine that keeps the columns' order: levels, stats and callbacks, with the tail of small levels
    mined directly (200,000 candidate words) or not at all."""
    import torch

    engm = import_module(pkg.__name__ + ".engine")
    syn = pkg.synthetic
    if data == "dense":
        n_rows, s, length = 30_011, 0.01, 4
        p = np.minimum(syn.dense_k2_probs(300, seed=2) * 2, 0.9)
        bv = syn.bernoulli_bitvecs(syn.bernoulli_thresholds(p), n_rows, seed=3)
        bv[7] = bv[8]
    else:
        from oracle import miner

        t = syn.plain_small(n_rows=20_000, n_items=300, seed=5)
        uniq, inv = np.unique(t.items, return_inverse=True)
        n_rows, s, length = t.n_rows, 0.003, None
        bv = miner.bitvecs_from_csr(t.indptr, inv.astype(np.int32), len(uniq), n_rows)
    dev = torch.from_numpy(np.ascontiguousarray(bv).view(np.int64)).cuda().view(torch.uint64)
    monkeypatch.setattr(engm, "DIRECT_WORDS", direct_words)
    monkeypatch.setattr(engm, "ORDER_WORDS", 0)
    plain, ordered = engm.Engine(), engm.Engine()
    plain.by_support = False
    calls = [[], []]
    a = plain.mine(dev, n_rows, s, length, level_callback=lambda *x: calls[0].append(x[:3]), **kw)
    b = ordered.mine(dev, n_rows, s, length, level_callback=lambda *x: calls[1].append(x[:3]), **kw)
    c = ordered.mine(dev, n_rows, s, length, **kw)
    assert len(a.levels) >= 2 and calls[0] == calls[1]
    for x in (b, c):
        assert [(t.k, t.n_candidates, t.n_frequent, t.n_groups) for t in x.stats] == \
            [(t.k, t.n_candidates, t.n_frequent, t.n_groups) for t in a.stats]
        assert len(x.levels) == len(a.levels)
        for lx, la in zip(x.levels, a.levels):
            assert torch.equal(lx.rows, la.rows) and torch.equal(lx.counts, la.counts)
    flushed = {}
    ordered.mine(dev, n_rows, s, length, keep_levels=False, on_level=lambda k, r, n: flushed.update({k: (r, n)}), **kw)
    for r, n in a.host_levels():
        assert np.array_equal(flushed[r.shape[1]][0], r) and np.array_equal(flushed[r.shape[1]][1], n)


@pytest.mark.parametrize("sizes", [[1, 1], [300, 40, 1], [20_000, 700, 0], [5, 17_000, 40_000]])
def test_levels_ordered_in_one_call(pkg, sizes):
    """etm_order_levels against etm_order_level and etm_group_totals of each level, and etm_frame_level of the results
    against numpy."""
    import torch

    lib = pkg.load_library()
    rng = np.random.default_rng(sum(sizes))
    n_items, k0 = 90, 3
    levels = [_level(rng, n, k0 + i, n_items)[:n] for i, n in enumerate(sizes)]
    sizes = [len(x) for x in levels]
    counts = [rng.integers(1, 10_000, n).astype(np.int32) for n in sizes]
    perm = rng.permutation(n_items).astype(np.int32)
    prev = np.unique(_level(rng, 500, k0 - 1, n_items), axis=0)
    rows_d = torch.from_numpy(np.concatenate([x.ravel() for x in levels])).cuda()
    counts_d, perm_d, prev_d = (torch.from_numpy(x).cuda() for x in (np.concatenate(counts), perm, prev))
    out_r, out_c = torch.empty_like(rows_d), torch.empty_like(counts_d)
    totals = torch.full((len(sizes), 2), -5, dtype=torch.int64, device="cuda")
    bits, need, one = 7, 1, ctypes.c_int64()
    for i, n in enumerate(sizes):
        assert lib.etm_order_level_bytes(n, k0 + i, bits, ctypes.byref(one)) == 0
        need = max(need, one.value)
    scratch = torch.empty(need, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    host_sizes = np.array(sizes, np.int64)
    assert lib.etm_order_levels(rows_d.data_ptr(), counts_d.data_ptr(), host_sizes.ctypes.data, len(sizes), k0,
                                perm_d.data_ptr(), bits, prev_d.data_ptr(), len(prev), out_r.data_ptr(),
                                out_c.data_ptr(), totals.data_ptr(), scratch.data_ptr(), need, stream) == 0, lib.etm_last_error()
    table = rng.integers(-2**62, 2**62, n_items)
    n, n_values = sum(sizes), out_r.numel()
    values, offsets = torch.empty(n_values, dtype=torch.int64).cuda(), torch.empty(n + 1, dtype=torch.int64).cuda()
    support, table_d = torch.empty(n, dtype=torch.float64).cuda(), torch.from_numpy(table).cuda()
    r = c = 0
    for i, (x, y) in enumerate(zip(levels, counts)):
        want = np.sort(perm[x], axis=1)
        at = np.lexsort(want.T[::-1])
        got = out_r[r:r + x.size].view(len(x), k0 + i)
        assert np.array_equal(got.cpu().numpy(), want[at]) and np.array_equal(out_c[c:c + len(x)].cpu().numpy(), y[at])
        if len(prev):
            runs = np.unique(prev[:, :-1], axis=0, return_counts=True)[1]
            assert totals[i].tolist() == [int((runs * (runs - 1) // 2).sum()), int((runs > 1).sum())]
        else:
            assert totals[i].tolist() == [0, 0]
        assert lib.etm_frame_level(out_r[r:].data_ptr(), out_c[c:].data_ptr(), len(x), k0 + i, table_d.data_ptr(), 12_347,
                                   c, r, values.data_ptr(), offsets.data_ptr(), support.data_ptr(), stream) == 0
        prev, r, c = want[at], r + x.size, c + len(x)
    assert np.array_equal(values.cpu().numpy(), table[out_r.cpu().numpy()])
    assert np.array_equal(support.cpu().numpy(), out_c.cpu().numpy().astype(np.float64) / 12_347)
    lens = np.concatenate([np.full(m, k0 + i) for i, m in enumerate(sizes)])
    assert np.array_equal(offsets.cpu().numpy(), np.concatenate([[0], np.cumsum(lens)]))
