"""Tables small enough for one launch, mined level by level all the same: the tensor cores, the projection and the
compaction on the sizes where their limits and their failures are tested."""

from __future__ import annotations

from importlib import import_module

import numpy as np
import pytest
from tests.conftest import case_input
from tests.helpers import digest_pairs, table_of

pytestmark = pytest.mark.gpu


@pytest.fixture
def engm(pkg):
    return import_module(pkg.__name__ + ".engine")


def _general(engm, **kw):
    eng = engm.Engine(**kw)
    eng.direct = False
    eng.profile_kernels = True
    return eng


def _names(eng):
    return {e[0] for e in eng._events}


def _dense(pkg, n_items):
    import torch

    syn = pkg.synthetic
    p = np.minimum(syn.dense_k2_probs(n_items, seed=9) * 3, 0.9)
    bv = syn.bernoulli_bitvecs(syn.bernoulli_thresholds(p), 20_000, seed=5)
    return torch.from_numpy(bv.view(np.int64)).cuda().view(torch.uint64)


def _same(a, b):
    assert len(a) == len(b) >= 3
    for (ra, ca), (rb, cb) in zip(a, b):
        assert np.array_equal(ra, rb) and np.array_equal(ca, cb)


@pytest.mark.parametrize("limit", [100, 256, 1000])
@pytest.mark.parametrize("name", ["dense_k2_small", "implication_infer", "deep_sparse_small"])
def test_groups_past_the_exact_row_limit(pkg, engm, golden_cases, monkeypatch, name, limit):
    """The Gram's exact row limit (2^24) lowered: longer groups, K=2 among them, are cut into parts that keep to it."""
    monkeypatch.setattr(engm, "TC_MAX_ROWS", limit)
    case = golden_cases[name]
    indptr, items, n_rows = case_input(pkg, case)
    eng = _general(engm)
    eng.k2_rows_max_r = eng.k3_rows_max_r = 0.0  # not from the rows
    got = pkg.apriori(table_of(indptr, items, n_rows), min_support=case["min_support"], max_length=case["max_length"],
                      use_gpu=True, prune_equal_support=case["prune_equal_support"],
                      use_generator_pruning=case["use_generator_pruning"], engine=eng, warn_complexity=False)
    assert digest_pairs(pkg.result_pairs(got, n_rows)) == case["digest"]
    assert "mine_direct" not in _names(eng) and "gram_tc" in _names(eng)


def test_dense_tables_on_the_tensor_cores_match_popcount(pkg, engm):
    dev = _dense(pkg, 400)
    pop, ten = _general(engm, method="popcount"), _general(engm, method="tensor")
    _same(pop.mine(dev, 20_000, 0.01, 3).host_levels(), ten.mine(dev, 20_000, 0.01, 3).host_levels())
    assert "gram_tc" in _names(ten) - _names(pop) and "mine_direct" not in _names(ten)


def test_exact_again_after_a_wait_gave_up(pkg, engm):
    lib = pkg.load_library()
    dev = _dense(pkg, 300)
    want = _general(engm, method="popcount").mine(dev, 20_000, 0.01, 3).host_levels()
    assert lib.etm_device_status(None) == 0
    try:
        for gram_ns, proj_ns in ((0, -1), (-1, 0)):
            assert lib.etm_set_wait_limits(gram_ns, proj_ns) == 0
            with pytest.raises(RuntimeError, match="bounded wait"):
                _general(engm, proj_rows=False).mine(dev, 20_000, 0.01, 3)
            assert lib.etm_device_status(None) == 0  # read and cleared by the engine
    finally:
        lib.etm_set_wait_limits(-1, -1)
    for kw in ({}, {"proj_rows": False}):
        _same(_general(engm, **kw).mine(dev, 20_000, 0.01, 3).host_levels(), want)


@pytest.mark.parametrize("limit", [1 << 24, 1000])
def test_no_room_for_the_blocked_columns_of_pairs(pkg, engm, monkeypatch, limit):
    """K=2 from the columns as they are: whole block pairs, or past their exact row limit the CUDA cores."""
    import torch

    dev = _dense(pkg, 300)
    want = _general(engm, method="popcount").mine(dev, 20_000, 0.01, 3).host_levels()
    monkeypatch.setattr(engm, "TC_MAX_ROWS", limit)
    eng = _general(engm)

    def refuse(*args):
        raise torch.OutOfMemoryError("no room")

    monkeypatch.setattr(eng, "_blocked_cols", refuse)
    _same(eng.mine(dev, 20_000, 0.01, 3).host_levels(), want)
    assert ("count_tiles" in _names(eng)) == (limit < 20_000)
