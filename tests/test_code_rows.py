"""The item coding's decisions on the host (no GPU needed)."""

from __future__ import annotations

from importlib import import_module

import numpy as np
import pytest


@pytest.mark.parametrize("ids", [[3, 2**63 + 5, 2**64 - 1], [2**63 - 1, 2**63, 2**63 + 1]])
def test_ids_on_the_host_are_left_alone(pkg, ids):
    """UInt64 ids, of too wide a span for the coding and of a narrow one: the caller's array keeps its values."""
    api = import_module(pkg.__name__ + ".api")
    flat = np.array(ids, np.uint64)
    indptr = np.array([0, 2, 3], np.int64)
    if int(flat.max()) - int(flat.min()) + 1 > api.CODE_SPAN_MAX:
        assert api._code_rows(indptr, flat, 2, 1, "cpu") is None
    else:
        with pytest.raises(RuntimeError, match="CUDA device"):
            api._code_rows(indptr, flat, 2, 1, "cpu")
    assert flat.tolist() == ids
