"""Block pairs that stop early and block pairs that run to their last row: the same levels."""

from __future__ import annotations

from importlib import import_module

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [{}, {"prune_equal_support": True}])
def test_a_mine_without_the_early_stop(pkg, monkeypatch, kw):
    import torch

    engm = import_module(pkg.__name__ + ".engine")
    syn = pkg.synthetic
    n_rows = 60_000
    p = np.minimum(syn.dense_k2_probs(500, seed=9), 0.9)
    bv = syn.bernoulli_bitvecs(syn.bernoulli_thresholds(p), n_rows, seed=5)
    dev = torch.from_numpy(bv.view(np.int64)).cuda().view(torch.uint64)
    monkeypatch.setattr(engm, "DIRECT_WORDS", 0)
    monkeypatch.setattr(engm, "ORDER_WORDS", 0)
    stops, runs = engm.Engine(), engm.Engine()
    runs.early_stop = False
    called = []
    lib = runs.lib

    class Library:
        def __getattr__(self, name):
            called.append(name)
            return getattr(lib, name)

    runs.lib = Library()
    a, b = stops.mine(dev, n_rows, 0.002, 3, **kw), runs.mine(dev, n_rows, 0.002, 3, **kw)
    assert "etm_count_tiles_tc_bound" not in called and any(n.startswith("etm_count_tiles_tc") for n in called)
    assert len(a.levels) == len(b.levels) == 2
    for x, y in zip(a.levels, b.levels):
        assert torch.equal(x.rows, y.rows) and torch.equal(x.counts, y.counts)
