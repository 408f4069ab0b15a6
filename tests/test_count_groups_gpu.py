"""etm_count_groups against a numpy recount: sizes around its 8-member tiles, one slab and several, every width that
has a prefix or none, dense counts and the fused threshold, with and without classes. Zero tolerance."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = np.array([2, 3, 4, 5, 6, 7, 8, 9, 10, 12, 13, 16, 17, 2, 24, 31], np.int64)


def _groups(width, seed):
    """Rows of one sorted level: a group of SIZES[g] members after each prefix, and one row between that has none."""
    rng = np.random.default_rng(seed)
    rows, first, n_cols = [], [], 48
    for g, m in enumerate(SIZES if width > 1 else [31]):
        prefix = [g] * min(1, width - 1) + list(range(20, 20 + max(0, width - 2)))
        first.append(len(rows))
        members = np.sort(rng.choice(np.arange(20 + max(0, width - 2), 20 + max(0, width - 2) + 31), int(m), False)) \
            if width > 1 else np.arange(m)
        rows += [prefix + [int(v)] for v in members]
    n_cols = max(max(r) for r in rows) + 1
    return np.array(rows, np.int32), np.array(first, np.int64), n_cols


@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("with_cls", [True, False])
@pytest.mark.parametrize("width,n_words", [(1, 1), (2, 1), (2, 33), (3, 64), (2, 2047), (4, 2048), (3, 2049),
                                           (6, 4097), (2, 10_001)])
def test_counts_match_a_recount(pkg, width, n_words, with_cls, fused):
    import torch

    lib = pkg.load_library()
    rows, first, n_cols = _groups(width, n_words)
    sizes = SIZES if width > 1 else np.array([31], np.int64)
    n = len(sizes)
    ld = (n_words + 31) // 32 * 32
    rng = np.random.default_rng(width)
    bv = np.zeros((n_cols, ld), np.uint64)
    bv[:, :n_words] = rng.integers(0, 2**63, size=(n_cols, n_words), dtype=np.int64).view(np.uint64)
    cand_off = np.zeros(n + 1, np.int64)
    np.cumsum(sizes * (sizes - 1) // 2, out=cand_off[1:])
    want = []
    for g in range(n):
        r = rows[first[g]:first[g] + sizes[g]]
        pre = np.bitwise_and.reduce(bv[r[0, :-1]], axis=0) if width > 1 else np.full(ld, 2**64 - 1, np.uint64)
        x = bv[r[:, -1]] & pre
        i, j = np.triu_indices(int(sizes[g]), 1)
        want.append(np.bitwise_count(x[i] & x[j]).sum(axis=1))
    want = np.concatenate(want).astype(np.int64)
    # The listed groups: every other one (and the first), the others keep their slots.
    listed = np.arange(0, n, 2, dtype=np.int64)
    m = sizes[listed]
    woff, toff = np.zeros(len(listed) + 1, np.int64), np.zeros(len(listed) + 1, np.int64)
    np.cumsum(m * (m - 1) // 2, out=woff[1:])
    nb = -(-m // 8)
    np.cumsum(nb * (nb + 1) // 2, out=toff[1:])
    cls = rng.integers(0, 3, len(want)).astype(np.uint8)
    mc = int(np.median(want))
    on = np.repeat(np.isin(np.arange(n), listed), sizes * (sizes - 1) // 2)
    if with_cls:
        on &= cls == 0
    if fused:
        on &= want >= mc
    expect = np.where(on, want, -3)

    def dev(a):
        return torch.from_numpy(np.ascontiguousarray(a)).cuda()

    d = [dev(a) for a in (bv.view(np.int64), rows, first, sizes.astype(np.int32), cand_off, listed, woff, toff, cls)]
    out = torch.full((len(want),), -3, dtype=torch.int32, device="cuda")
    bits = torch.zeros(len(want) // 32 + 2, dtype=torch.int32, device="cuda")
    partial = torch.full((int(woff[-1]),), 9, dtype=torch.int32, device="cuda") if n_words > 2048 else None
    st = lib.etm_count_groups(
        d[0].data_ptr(), ld, n_words, d[1].data_ptr(), width, d[2].data_ptr(), d[3].data_ptr(), d[4].data_ptr(),
        d[5].data_ptr(), d[6].data_ptr(), d[7].data_ptr(), len(listed), int(woff[-1]), int(toff[-1]), 0,
        d[8].data_ptr() if with_cls else None, mc, out.data_ptr(), bits.data_ptr() if fused else None,
        None if partial is None else partial.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert st == 0, lib.etm_last_error()
    assert np.array_equal(out.cpu().numpy(), expect)
    got_bits = np.unpackbits(bits.cpu().numpy().view(np.uint8), bitorder="little")[:len(want)]
    assert np.array_equal(got_bits.astype(bool), on if fused else np.zeros(len(want), bool))


def test_several_slabs_need_the_partial_counts(pkg):
    lib = pkg.load_library()
    assert lib.etm_count_groups(None, 2080, 2049, None, 2, None, None, None, None, None, None, 1, 1, 1, 0, None, 1,
                                None, None, None, None) == 1
