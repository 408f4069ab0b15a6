"""etm_order_level on levels whose rows share their first items: the keys' leading bits tell nothing apart."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N_ITEMS = 2000


def _shared_prefix(rng, n, k):
    """n rows of k items, the first k - 2 of all rows alike."""
    pairs = np.stack(np.triu_indices(400, 1), 1)[:n] + k
    return rng.permutation(np.concatenate([np.tile(np.arange(k - 2), (n, 1)), pairs], axis=1)).astype(np.int32)


def _spread(rng, n, k):
    rows = np.sort(rng.integers(0, N_ITEMS, (2 * n + 64, k)), axis=1)
    return rng.permutation(np.unique(rows[(np.diff(rows, axis=1) > 0).all(axis=1)], axis=0))[:n].astype(np.int32)


def _order(lib, rows):
    """(rows, counts, the fastest of a few runs in us)."""
    import torch

    n, k = rows.shape
    bits = (N_ITEMS - 1).bit_length()
    need = ctypes.c_int64()
    assert lib.etm_order_level_bytes(n, k, bits, ctypes.byref(need)) == 0
    d = torch.from_numpy(rows).cuda()
    counts, perm = torch.arange(n, dtype=torch.int32, device="cuda"), torch.arange(N_ITEMS, dtype=torch.int32, device="cuda")
    out, out_c = torch.empty_like(d), torch.empty_like(counts)
    scratch = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    times = []
    for _ in range(5):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        assert lib.etm_order_level(d.data_ptr(), counts.data_ptr(), n, k, perm.data_ptr(), bits, out.data_ptr(),
                                   out_c.data_ptr(), scratch.data_ptr(), need.value,
                                   torch.cuda.current_stream().cuda_stream) == 0, lib.etm_last_error()
        e1.record()
        e1.synchronize()
        times.append(e0.elapsed_time(e1) * 1e3)
    return out.cpu().numpy(), out_c.cpu().numpy(), min(times)


@pytest.mark.parametrize("k", [3, 4, 9, 23])
@pytest.mark.parametrize("n", [2049, 4096, 6145, 40_000, 65_535, 65_536])
def test_rows_with_shared_first_items(pkg, n, k):
    lib = pkg.load_library()
    rng = np.random.default_rng(n + k)
    rows = _shared_prefix(rng, n, k)
    got, counts, us = _order(lib, rows)
    at = np.lexsort(rows.T[::-1])
    assert np.array_equal(got, rows[at]) and np.array_equal(counts, at)
    if n >= 40_000:
        # Rows alike in a word take a second look at every comparison, not one at all the others.
        spread = _spread(rng, n, k)
        got, counts, base = _order(lib, spread)
        at = np.lexsort(spread.T[::-1])
        assert np.array_equal(got, spread[at]) and np.array_equal(counts, at)
        assert us < 8 * base
