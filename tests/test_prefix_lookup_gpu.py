"""etm_prefix_lookup and the segment offsets against numpy, and the decoding of survivors from the bitmask for groups of
every size around a word. Zero tolerance."""

from __future__ import annotations

from importlib import import_module

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [2, 3, 5])
def test_prefixes_find_their_rows(pkg, width):
    import torch

    lib = pkg.load_library()
    rng = np.random.default_rng(width)
    prev = np.unique(np.sort(rng.integers(0, 60, (700, width - 1)), axis=1), axis=0).astype(np.int32)
    counts = rng.integers(1, 10**6, len(prev)).astype(np.int32)
    pick = rng.integers(0, len(prev), 90)
    rows = np.concatenate([prev[pick], np.full((90, 1), 99, np.int32)], axis=1)
    rows[::7, 0] = 77  # no row of the level
    first = np.arange(90, dtype=np.int64)
    want = np.where(np.arange(90) % 7 == 0, -1, counts[pick])
    d = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (rows, first, prev, counts)]
    out = torch.empty(90, dtype=torch.int64, device="cuda")
    assert lib.etm_prefix_lookup(d[0].data_ptr(), width, d[1].data_ptr(), 90, d[2].data_ptr(), d[3].data_ptr(), len(prev),
                                 out.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0, lib.etm_last_error()
    assert np.array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("n_words", [1, 1023, 1024, 1025, 33 * 1024 + 7])
def test_segment_offsets(pkg, n_words):
    """Few groups over many segments and many groups over one: the padded words of every segment's prefix rows."""
    import torch

    lib = pkg.load_library()
    rng = np.random.default_rng(n_words)
    n_g = 5 if n_words > 5000 else 300
    ld = (n_words + 31) // 32 * 32
    bv = np.zeros((n_g, ld), np.uint64)
    bv[:, :n_words] = rng.integers(0, 2**63, (n_g, n_words), dtype=np.int64).view(np.uint64)
    bv[0] = 0
    rows = np.stack([np.arange(n_g), (np.arange(n_g) + 1) % n_g, np.full(n_g, n_g)], 1).astype(np.int32)
    n_seg = -(-n_words // 1024)
    d = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (
        bv.view(np.int64), rows, np.arange(n_g, dtype=np.int64), np.arange(n_g, dtype=np.int64))]
    off = torch.empty((n_g, n_seg + 1), dtype=torch.int64, device="cuda")
    words = torch.empty(n_g, dtype=torch.int64, device="cuda")
    assert lib.etm_prefix_segments(d[0].data_ptr(), ld, n_words, d[1].data_ptr(), 3, d[2].data_ptr(), d[3].data_ptr(), n_g,
                                   off.data_ptr(), words.data_ptr(), None, 0,
                                   torch.cuda.current_stream().cuda_stream) == 0, lib.etm_last_error()
    both = bv[rows[:, 0]] & bv[rows[:, 1]]
    pad = np.zeros((n_g, n_seg * 1024), np.uint64)
    pad[:, :ld] = both[:, :n_seg * 1024]
    per = np.bitwise_count(pad.reshape(n_g, n_seg, 1024)).astype(np.int64).sum(axis=2)
    want = np.zeros((n_g, n_seg + 1), np.int64)
    np.cumsum(((per + 63) // 64 + 3) // 4 * 4, axis=1, out=want[:, 1:])
    assert np.array_equal(off.cpu().numpy(), want) and np.array_equal(words.cpu().numpy(), want[:, -1])


@pytest.mark.parametrize("density", [0.0005, 0.3, 1.0])
@pytest.mark.parametrize("sizes", ["pairs", "mixed", "one", "wide"])
def test_bitmask_survivors_decode_in_order(pkg, sizes, density):
    """Groups of two (32 of them in a word), of mixed sizes, one of 3,000, and thousands of candidates past a tile."""
    import torch

    lib = pkg.load_library()
    engm = import_module(pkg.__name__ + ".engine")
    rng = np.random.default_rng(len(sizes))
    m = {"pairs": np.full(5000, 2), "mixed": rng.integers(2, 70, 900), "one": np.array([3000]),
         "wide": np.concatenate([np.full(100, 2), [900], np.full(40, 3), [1200]])}[sizes].astype(np.int64)
    rows = np.stack([np.repeat(np.arange(len(m)), m), np.concatenate([np.arange(x) for x in m])], 1).astype(np.int32)
    dev = torch.device("cuda")
    level = engm.Level(torch.from_numpy(rows).to(dev), torch.ones(len(rows), dtype=torch.int32, device=dev))
    G, total, gf, gs, co = engm.Engine().groups(level)
    assert G == len(m) and total == int((m * (m - 1) // 2).sum())
    keep = rng.random(total) < density
    counts = rng.integers(1, 10**6, total).astype(np.int32)
    bits = np.zeros(-(-total // 32) * 32, bool)
    bits[:total] = keep
    surv = torch.from_numpy(np.packbits(bits, bitorder="little").view(np.int32).copy()).to(dev)
    first = np.cumsum(m) - m
    i = np.concatenate([np.triu_indices(int(x), 1)[0] + f for x, f in zip(m, first)])
    j = np.concatenate([np.triu_indices(int(x), 1)[1] + f for x, f in zip(m, first)])
    want = np.concatenate([rows[i], rows[j][:, 1:]], 1)[keep]
    cap = max(1, int(keep.sum()))
    out_r = torch.empty((cap, 3), dtype=torch.int32, device=dev)
    out_c = torch.empty(cap, dtype=torch.int32, device=dev)
    acc = torch.zeros(1, dtype=torch.int64, device=dev)
    ws = torch.empty(engm.scan_words(len(bits) // 32), dtype=torch.int64, device=dev)
    c = torch.from_numpy(counts).to(dev)
    st = lib.etm_level_compact_bits(surv.data_ptr(), c.data_ptr(), total, level.rows.data_ptr(), 2, gf.data_ptr(),
                                    gs.data_ptr(), co.data_ptr(), 0, G, out_r.data_ptr(), out_c.data_ptr(), cap,
                                    acc.data_ptr(), ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
    assert st == 0, lib.etm_last_error()
    n = int(acc.item())
    assert n == int(keep.sum())
    assert np.array_equal(out_r.cpu().numpy()[:n], want) and np.array_equal(out_c.cpu().numpy()[:n], counts[keep])
