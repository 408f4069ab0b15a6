"""The coding of any transactions (unsorted rows, repeated ids, UInt64 ids) without a device-wide sort, against numpy and the
sorting path. Zero tolerance."""

from __future__ import annotations

from importlib import import_module

import numpy as np
import pytest

from tests.helpers import table_of

pytestmark = pytest.mark.gpu


def _rows(rng, lens, n_ids):
    indptr = np.zeros(len(lens) + 1, np.int64)
    np.cumsum(lens, out=indptr[1:])
    return indptr, rng.integers(0, n_ids, int(indptr[-1])).astype(np.int64)


LENS = [[0, 1, 2, 31, 32, 33, 0, 63, 64, 65, 500, 1], [2048, 3, 0, 1025, 40], [7] * 300]


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("n_ids", [3, 50, 100_000])
def test_rows_are_sorted_in_place(pkg, lens, n_ids):
    import torch

    lib = pkg.load_library()
    indptr, codes = _rows(np.random.default_rng(n_ids), lens, n_ids)
    rp, c = torch.from_numpy(indptr).cuda(), torch.from_numpy(codes.astype(np.int32)).cuda()
    st = torch.full((1,), 7, dtype=torch.int32, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    assert lib.etm_sort_rows(rp.data_ptr(), len(lens), c.data_ptr(), st.data_ptr(), stream) == 0, lib.etm_last_error()
    want = []
    for r in range(len(lens)):
        u = np.unique(codes[indptr[r]:indptr[r + 1]])
        want += u.tolist() + [-1] * (lens[r] - len(u))
    assert c.cpu().tolist() == want and int(st.item()) == 0
    lut = np.where(np.arange(n_ids) % 3 == 0, -1, np.arange(n_ids)).astype(np.int32)
    out = torch.empty(2, dtype=torch.int64, device="cuda")
    ld = torch.from_numpy(lut).cuda()
    assert lib.etm_row_pairs(rp.data_ptr(), c.data_ptr(), len(lens), ld.data_ptr(), n_ids, out.data_ptr(), stream) == 0
    kept = [sum(1 for x in want[indptr[r]:indptr[r + 1]] if x >= 0 and x % 3) for r in range(len(lens))]
    assert out.tolist() == [sum(n * (n - 1) // 2 for n in kept), max(lens)]


def test_a_row_too_long_to_sort_is_reported_and_kept(pkg):
    import torch

    lib = pkg.load_library()
    indptr, codes = _rows(np.random.default_rng(1), [5, 2049], 10)
    rp, c = torch.from_numpy(indptr).cuda(), torch.from_numpy(codes.astype(np.int32)).cuda()
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert lib.etm_sort_rows(rp.data_ptr(), 2, c.data_ptr(), st.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    assert int(st.item()) == 1 and c[5:].cpu().tolist() == codes[5:].tolist()


@pytest.mark.parametrize("ids", ["int64", "uint64"])
@pytest.mark.parametrize("mc", [1, 3])
@pytest.mark.parametrize("lens", LENS)
def test_coding_matches_the_sorting_path(pkg, lens, mc, ids):
    import torch

    api = import_module(pkg.__name__ + ".api")
    rng = np.random.default_rng(mc)
    indptr, flat = _rows(rng, lens, 90)
    if ids == "uint64":
        flat = flat.astype(np.uint64) * np.uint64(1000) + np.uint64(2**63 - 40_000)  # both sides of 2^63
    else:
        flat = flat * 1000 - 40_000
    n = len(lens)
    got = api._code_rows(indptr, flat, n, mc, torch.device("cuda"))
    row_ptr, cols, items, row_len, support = api._frequent_csr_device(indptr, flat, n, mc, "cuda")
    assert got.items.dtype == items.dtype and np.array_equal(got.items, items)
    assert np.array_equal(got.support, support)
    assert got.row_len == float((row_len * (row_len - 1) // 2).sum())
    col_of, codes, rp = got.col_of.cpu().numpy(), got.codes.cpu().numpy(), row_ptr.cpu().numpy()
    for r in range(n):
        c = codes[indptr[r]:indptr[r + 1]]
        mine = [int(col_of[x]) for x in c if x >= 0 and col_of[x] >= 0]
        assert mine == cols[rp[r]:rp[r + 1]].cpu().tolist()


@pytest.mark.parametrize("shape", ["rows", "span"])
def test_mines_of_recorded_rows(pkg, shape):
    """Unsorted rows with repeats, mined as their sorted, repeat-free twins; rows past the sort's length and ids past the
    bitmap's span still take the sorting path."""
    syn = pkg.synthetic
    t = syn.plain_small(n_rows=4000, n_items=200, seed=2)
    rng = np.random.default_rng(0)
    rows = []
    for r in range(t.n_rows):
        x = t.items[t.indptr[r]:t.indptr[r + 1]]
        rows.append(rng.permutation(np.concatenate([x, rng.choice(x, 2)])))
    if shape == "rows":
        rows[17] = np.concatenate([rows[17], np.repeat(rows[17], 400)])
    indptr = np.zeros(len(rows) + 1, np.int64)
    np.cumsum([len(x) for x in rows], out=indptr[1:])
    flat = np.concatenate(rows)
    items = t.items
    if shape == "span":
        flat, items = flat * (1 << 22), items * (1 << 22)
    kw = dict(min_support=0.01, use_gpu=True, warn_complexity=False, max_length=6)
    want = pkg.result_pairs(pkg.apriori(table_of(t.indptr, items, t.n_rows), **kw), t.n_rows)
    got = pkg.result_pairs(pkg.apriori(table_of(indptr, flat, t.n_rows), **kw), t.n_rows)
    assert len(want) > 100 and got == want


@pytest.mark.parametrize("n_ids", [12_288, 12_289, 55_296, 55_297])
@pytest.mark.parametrize("nnz", [1000, 9_000_000])
def test_histogram_bins_around_its_forms(pkg, n_ids, nnz):
    import torch

    lib = pkg.load_library()
    codes = torch.randint(-1, n_ids + 1, (nnz,), dtype=torch.int32, device="cuda")
    out = torch.empty(n_ids, dtype=torch.int64, device="cuda")
    assert lib.etm_code_histogram(codes.data_ptr(), nnz, n_ids, out.data_ptr(),
                                  torch.cuda.current_stream().cuda_stream) == 0, lib.etm_last_error()
    ok = codes[(codes >= 0) & (codes < n_ids)].long()
    assert torch.equal(out, torch.bincount(ok, minlength=n_ids))


@pytest.mark.parametrize("n", [1, 31, 4096, 4097, 70_001])
def test_id_bounds_and_code_columns(pkg, n):
    """The bounds of the ids over the whole range, and the frequent codes' places."""
    import torch

    lib = pkg.load_library()
    rng = np.random.default_rng(n)
    stream = torch.cuda.current_stream().cuda_stream
    for lo, hi in ((-2**63, 2**63 - 1), (-5, 3), (7, 7)):
        ids = rng.integers(lo, hi, n, endpoint=True)
        d, out = torch.from_numpy(ids).cuda(), torch.empty(2, dtype=torch.int64, device="cuda")
        assert lib.etm_id_range(d.data_ptr(), n, out.data_ptr(), stream) == 0
        top, low = (int(x) for x in out.cpu().numpy().view(np.uint64))
        assert (top - 2**63, 2**64 - 1 - low - 2**63) == (int(ids.max()), int(ids.min()))
    counts = rng.integers(0, 20, n)
    d = torch.from_numpy(counts).cuda()
    col = torch.full((n,), 9, dtype=torch.int32, device="cuda")
    ws = torch.empty(n // 4096 + 3, dtype=torch.int64, device="cuda")
    for mc in (1, 10, 30):
        assert lib.etm_code_columns(d.data_ptr(), n, mc, col.data_ptr(), ws.data_ptr(), ws.numel(), stream) == 0
        keep = counts >= mc
        assert np.array_equal(col.cpu().numpy(), np.where(keep, np.cumsum(keep) - 1, -1))
