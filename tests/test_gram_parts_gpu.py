"""The packed e2m1 Gram over blocked rows cut along its rows, and the blocked copy of the columns it reads at K=2.
Integer results: zero tolerance."""

from __future__ import annotations

from importlib import import_module

import numpy as np
import pytest

from tests.test_tensor_gpu import _gram_groups


@pytest.mark.gpu
@pytest.mark.parametrize("with_counter", [True, False])
@pytest.mark.parametrize("with_cls", [True, False])
@pytest.mark.parametrize("parts", [[1] * 7, [2, 1, 1, 3, 2, 1, 2], [16, 1, 1, 33, 5, 1, 2]])
def test_parts_add_up_to_the_whole_counts(pkg, parts, with_cls, with_counter):
    """Parts of one stage, empty parts (more parts than stages) and whole pairs in one launch; candidates of
    another class than COUNT keep what their slot held."""
    import torch

    lib = pkg.load_library()
    t, d, want, n_work, _ = _gram_groups(lib, 4, blocked=True)
    size = d["size"].cpu().numpy().astype(np.int64)
    nb = -(-size // t)
    p = np.array(parts, np.int64)
    off = np.zeros(n_work + 1, np.int64)
    np.cumsum(nb * (nb + 1) // 2 * p, out=off[1:])
    wo, pd = torch.from_numpy(off).cuda(), torch.from_numpy(p).cuda()
    cls = np.random.default_rng(3).integers(0, 3, len(want)).astype(np.uint8) if with_cls else None
    cls_d = torch.from_numpy(cls).cuda() if with_cls else None
    out = torch.zeros(len(want), dtype=torch.int32, device="cuda")
    if with_cls:
        out[cls_d != 0] = -7
        want = np.where(cls == 0, want, -7)
    counter = torch.zeros(1, dtype=torch.int64, device="cuda") if with_counter else None
    st = lib.etm_count_tiles_tc_parts(
        d["buf"].data_ptr(), d["cbase"].data_ptr(), d["cwords"].data_ptr(), d["cld"].data_ptr(), d["size"].data_ptr(),
        d["cand_off"].data_ptr(), d["wg"].data_ptr(), wo.data_ptr(), pd.data_ptr(), n_work, int(off[-1]), 0,
        cls_d.data_ptr() if with_cls else None, out.data_ptr(), counter.data_ptr() if with_counter else None,
        torch.cuda.current_stream().cuda_stream)
    assert st == 0, lib.etm_last_error()
    torch.cuda.synchronize()
    assert lib.etm_device_status(torch.cuda.current_stream().cuda_stream) == 0
    assert np.array_equal(out.cpu().numpy(), want)


@pytest.mark.gpu
@pytest.mark.parametrize("n_cols,ld", [(1, 32), (7, 64), (8, 32), (239, 96), (240, 1024), (241, 1056), (500, 2080)])
def test_blocked_columns_hold_every_word_at_its_place(pkg, n_cols, ld):
    import torch

    lib = pkg.load_library()
    blk = 240
    x = np.random.default_rng(n_cols).integers(-2**63, 2**63 - 1, size=(n_cols, ld), dtype=np.int64)
    out = torch.full((-(-n_cols // blk) * blk * ld,), 5, dtype=torch.int64, device="cuda")
    src = torch.from_numpy(x).cuda()
    assert lib.etm_block_cols(src.data_ptr(), ld, n_cols, blk, out.data_ptr(),
                              torch.cuda.current_stream().cuda_stream) == 0, lib.etm_last_error()
    j, w = np.arange(n_cols)[:, None], np.arange(ld)[None, :]
    at = (j // blk) * ld * blk + (w // 4) * 4 * blk + (w // 2 % 2) * 2 * blk + (j % blk) * 2 + w % 2
    want = np.full(out.numel(), 5, np.int64)
    want[at] = x
    assert np.array_equal(out.cpu().numpy(), want)


@pytest.mark.gpu
@pytest.mark.parametrize("n_rows,n_items", [(70_000, 17), (70_001, 130), (200_003, 241)])
def test_cut_levels_match_the_popcount_engine(pkg, n_rows, n_items):
    """Few block pairs over many rows (K=2 and K=3 cut into parts), with and without inference."""
    import torch

    engm = import_module(pkg.__name__ + ".engine")
    syn = pkg.synthetic
    p = np.minimum(syn.dense_k2_probs(n_items, seed=4) * 3, 0.9)
    bv = syn.bernoulli_bitvecs(syn.bernoulli_thresholds(p), n_rows, seed=6)
    dev = torch.from_numpy(bv.view(np.int64)).cuda().view(torch.uint64)
    for infer in (False, True):
        a = engm.Engine(method="popcount").mine(dev, n_rows, 0.02, 3, use_generator_pruning=infer).host_levels()
        b = engm.Engine(small_group=4).mine(dev, n_rows, 0.02, 3, use_generator_pruning=infer).host_levels()
        assert len(a) == len(b) == 3
        for (ra, ca), (rb, cb) in zip(a, b):
            assert np.array_equal(ra, rb) and np.array_equal(ca, cb)


def test_part_planning(pkg):
    engm = import_module(pkg.__name__ + ".engine")
    # One long pair: a quarter of the SM's share each, never shorter than GRAM_MIN_STAGES.
    assert engm.gram_parts([1], [235], 152).tolist() == [10]
    assert engm.gram_parts([3], [78125], 152)[0] == -(-78125 // -(-3 * 78125 // 608))
    # Many pairs of like length stay whole.
    assert engm.gram_parts(np.full(4000, 50), np.full(4000, 300), 152).max() == 1
    # A part holds at most 2^24 rows.
    assert engm.gram_parts([10**6], [1 << 17], 152)[0] == 2
